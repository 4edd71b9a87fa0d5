"""When an autograd function may run as a plain call."""
import subprocess
import sys
from pathlib import Path

import pytest
import torch
from torch.autograd import forward_ad

from aeris_gb_b200.models import fused


def test_plain_only_where_nothing_is_recorded():
    assert fused.recorded()
    with torch.no_grad():
        assert not fused.recorded()
        with forward_ad.dual_level():
            assert fused.recorded()
        seen = []
        torch.func.vmap(lambda t: (seen.append(fused.recorded()), t)[1])(torch.zeros(2))
        torch.jit.trace(lambda t: (seen.append(fused.recorded()), t + 1)[1], torch.zeros(2), check_trace=False)
        assert seen == [True, True]


@pytest.mark.parametrize("name", ["torch.autograd.forward_ad._current_level", "torch._C._are_functorch_transforms_active",
                                  "torch._C._get_tracing_state"])
def test_without_a_private_name_everything_counts_as_recorded(name):
    """The names are looked up at import: a process of its own, from which the name is gone first."""
    code = (f"import torch; del {name}\n" "from aeris_gb_b200.models import fused\n"
            "torch._C._set_grad_enabled(False)\n" "assert fused.recorded()\n")
    r = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).parent.parent, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-500:]
