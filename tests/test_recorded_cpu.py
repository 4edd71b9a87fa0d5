"""When an autograd function may run as a plain call."""
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


@pytest.mark.parametrize("owner,name", [(forward_ad, "_current_level"), (torch._C, "_are_functorch_transforms_active"),
                                        (torch._C, "_get_tracing_state")])
def test_without_a_private_name_everything_counts_as_recorded(owner, name, monkeypatch):
    monkeypatch.delattr(owner, name)
    try:
        with torch.no_grad():
            assert fused.recorded()
    finally:
        monkeypatch.undo()
