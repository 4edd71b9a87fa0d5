// All kernels of one transformer block, forward or backward, issued by one call.
//
// A block is 7 launches forward and about 20 backward per chunk and sample. Issued one by one from Python each costs the
// host 10-20 us (argument objects, views, checks), which is longer than most of them run on small models; here a launch
// costs what the driver takes for it.
#include <stdint.h>

#include "api.h"
#include "gemm_epilogue.cuh"

using namespace aeris;

namespace {

typedef __nv_bfloat16 bf16;

// Counts launches and keeps the first error: the code of the entry point that refused, less 1000 times its place.
struct Run {
  int launches = 0, rc = 0;
  bool operator()(int where, int code, int kernels = 1) {
    launches += kernels;
    if (code != 0) rc = code - 1000 * where;
    return code == 0;
  }
  int result() const { return rc ? rc : launches; }
};

template <typename T>
T* at(void* base, long long rows, long long pitch) {
  return base ? reinterpret_cast<T*>(base) + rows * pitch : nullptr;
}
template <typename T>
const T* at(const void* base, long long rows, long long pitch) {
  return base ? reinterpret_cast<const T*>(base) + rows * pitch : nullptr;
}

// C (op)= A B^T over row-major operands without gaps: `at` / `bt`: stored transposed.
struct Gemm {
  const AerisBlock& b;
  int operator()(const void* A, bool a_t, const void* B, bool b_t, void* C, int M, int N, int K, int epi, int ldc,
                 const void* resid = nullptr, int ldr = 0, const float* gate = nullptr, int rows_per_gate = 0,
                 void* aux = nullptr, int ld_aux = 0, int k_splits = 1) const {
    const int f = epi == EPI_SWIGLU || epi == EPI_SWIGLU_BOTH ? N / 2 : epi == EPI_SWIGLU_BWD ? N : 0;
    return aeris_gemm_auto(A, B, C, M, N, K, a_t ? M : K, b_t ? N : K, ldc, a_t, b_t, epi, resid, ldr, gate, rows_per_gate,
                           static_cast<int>(b.mod_sample), aux, ld_aux, f, k_splits, 0, b.two_cta, b.status, b.stream);
  }
};

struct Vectors {
  const float *shift1, *scale1, *gate1, *shift2, *scale2, *gate2;
};
Vectors vectors(const AerisBlock& b, int sample) {
  const float* m = b.mod + static_cast<long long>(sample) * b.mod_sample;
  return {m, m + b.mod_vec, m + 2 * b.mod_vec, m + 3 * b.mod_vec, m + 4 * b.mod_vec, m + 5 * b.mod_vec};
}

struct Chunk {
  bf16 *h1, *qkv, *o, *x1, *h2, *act, *u;
  float* lse;
};
// Where the internals of the chunk that starts at row `r0` live: full-size buffers or chunk workspaces.
Chunk chunk(const AerisBlock& b, long long r0) {
  const long long r = b.kept ? r0 : 0;
  const int HD = b.heads * b.head_dim;
  return {at<bf16>(b.h1, r, b.D),  at<bf16>(b.qkv, r, 3 * HD), at<bf16>(b.o, r, HD),       at<bf16>(b.x1, r, b.D),
          at<bf16>(b.h2, r, b.D),  at<bf16>(b.act, r, b.F),    at<bf16>(b.u, r, 2 * b.F),  at<float>(b.lse, r, b.heads)};
}

bool modnorm(const AerisBlock& b, Run& run, int where, const bf16* x, const uint32_t* table, bf16* x_out,
             const float* scale, const float* shift, const void* w, bf16* h, int nb, int rows) {
  const void* gx = table ? nullptr : x;
  if (nb == 1)
    return run(where, aeris_modnorm_fwd(gx, table, b.peers, b.n_peers, x_out, scale, shift, w, h, rows, b.D, b.mode, b.eps,
                                        nullptr, nullptr, b.stream));
  return run(where, aeris_modnorm_fwd_batch(gx, table, b.peers, b.n_peers, x_out, scale, shift,
                                            static_cast<int>(b.mod_sample), w, h, nb, rows / nb, b.D, b.mode, b.eps, nullptr,
                                            nullptr, b.stream));
}

bool rope(const AerisBlock& b, Run& run, int where, bf16* qkv, int rows, int inverse) {
  return !b.rope_cos ||
         run(where, aeris_rope_qk(qkv, b.rope_cos, b.rope_sin, rows, b.L, b.heads, b.head_dim, inverse, b.stream));
}

// First half of a chunk: h1 = modulated norm of x, q|k|v, attention, x1 = x + g1 * (o wo^T). `table`: x is gathered on the
// way (see aeris_modnorm_fwd).
bool attention_half(const AerisBlock& b, Run& run, const Chunk& c, const Vectors& v, bf16* x, const uint32_t* table, int nw,
                    int nb) {
  const Gemm gemm{b};
  const int n = nw * b.L, HD = b.heads * b.head_dim;
  return modnorm(b, run, 1, x, table, table ? x : nullptr, v.scale1, v.shift1, b.wn1, c.h1, nb, n) &&
         run(2, gemm(c.h1, false, b.wqkv, false, c.qkv, n, 3 * HD, b.D, EPI_STORE, 3 * HD)) &&
         rope(b, run, 3, c.qkv, n, 0) &&
         run(4, aeris_attn_fwd(c.qkv, 3 * HD, 0, c.qkv, 3 * HD, HD, c.qkv, 3 * HD, 2 * HD, c.o, HD, c.lse, nw, b.L, b.heads,
                               b.head_dim, b.scale, b.status, b.stream)) &&
         run(5, gemm(c.o, false, b.wo, false, c.x1, n, b.D, HD, EPI_GATE_RESID, b.D, x, b.D, v.gate1, n / nb));
}

// body(first row, windows) for every chunk of a sample, until one fails
template <typename F>
bool for_chunks(const AerisBlock& b, int sample, F&& body) {
  for (int w0 = 0; w0 < b.n_win; w0 += b.step) {
    const int nw = b.n_win - w0 < b.step ? b.n_win - w0 : b.step;
    if (!body((static_cast<long long>(sample) * b.n_win + w0) * b.L, nw)) return false;
  }
  return true;
}

}  // namespace

extern "C" int aeris_block_forward(const AerisBlock* pb) {
  const AerisBlock& b = *pb;
  if (b.step <= 0) return -1;        // chunks of no windows never end
  const Gemm gemm{b};
  Run run;
  auto body = [&](int sample, int nb, long long r0, int nw) {
    const Vectors v = vectors(b, sample);
    const Chunk c = chunk(b, r0);
    const int n = nw * b.L;
    bf16 *x = at<bf16>(b.x, r0, b.D), *y = at<bf16>(b.y, r0, b.D);
    return attention_half(b, run, c, v, x, b.table ? b.table + r0 : nullptr, nw, nb) &&
           modnorm(b, run, 6, c.x1, nullptr, nullptr, v.scale2, v.shift2, b.wn2, c.h2, nb, n) &&
           run(7, b.kept ? gemm(c.h2, false, b.w1, false, c.act, n, 2 * b.F, b.D, EPI_SWIGLU_BOTH, b.F, nullptr, 0, nullptr,
                                0, c.u, 2 * b.F)
                         : gemm(c.h2, false, b.w1, false, c.act, n, 2 * b.F, b.D, EPI_SWIGLU, b.F)) &&
           run(8, gemm(c.act, false, b.w2, false, y, n, b.D, b.F, EPI_GATE_RESID, b.D, c.x1, b.D, v.gate2, n / nb));
  };
  if (b.merged) {
    body(0, b.batch, 0, b.batch * b.n_win);
  } else {
    for (int s = 0; s < b.batch; ++s)
      if (!for_chunks(b, s, [&](long long r0, int nw) { return body(s, 1, r0, nw); })) break;
  }
  return run.result();
}

// The whole trunk of a network evaluation. A sampler's evaluations differ in the modulation vectors only: `mod_offset`
// elements further on in every block's.
extern "C" int aeris_blocks_forward(const AerisBlock* blocks, int n, long long mod_offset, void* stream) {
  int launches = 0;
  for (int i = 0; i < n; ++i) {
    AerisBlock b = blocks[i];
    b.mod += mod_offset;
    b.stream = stream;
    const int rc = aeris_block_forward(&b);
    if (rc < 0) return rc;
    launches += rc;
  }
  return launches;
}

extern "C" int aeris_block_backward(const AerisBlock* pb, const AerisBlockGrad* pg) {
  const AerisBlock& b = *pb;
  const AerisBlockGrad& g = *pg;
  if (b.step <= 0) return -1;
  const Gemm gemm{b};
  const int D = b.D, F = b.F, HD = b.heads * b.head_dim;
  Run run;
  for (int s = 0; s < b.batch; ++s) {
    const Vectors v = vectors(b, s);
    float* dm = g.dmod + static_cast<long long>(s) * 6 * D;      // shift1, scale1, gate1, shift2, scale2, gate2
    // G2 = dy^T act and Go = dx1^T o are the ungated gradients of w2 and wo for one sample
    if (!run(10, aeris_gate_prepare(b.w2, v.gate2, g.w2g, g.G2, F, b.wo, v.gate1, g.wog, g.Go, HD, D, dm, 6 * D, b.stream)))
      break;
    const bool ok = for_chunks(b, s, [&](long long r0, int nw) {
      const Chunk c = chunk(b, r0);
      const int n = nw * b.L, slices = -4 * ((nw + b.slice_windows - 1) / b.slice_windows);
      bf16 *x = at<bf16>(b.x, r0, D), *dx = at<bf16>(g.dx, r0, D);
      const bf16* dy = at<bf16>(g.dy, r0, D);
      bf16* u = b.kept ? c.u : reinterpret_cast<bf16*>(g.du);
      if (!b.kept &&
          !(attention_half(b, run, c, v, x, nullptr, nw, 1) &&
            modnorm(b, run, 6, c.x1, nullptr, nullptr, v.scale2, v.shift2, b.wn2, c.h2, 1, n) &&
            run(7, gemm(c.h2, false, b.w1, false, c.act, n, 2 * F, D, EPI_SWIGLU_BOTH, F, nullptr, 0, nullptr, 0, u,
                        2 * F))))
        return false;
      auto wgrad = [&](int where, const void* dout, int M, const void* in, int N, float* G) {
        return run(where, gemm(dout, true, in, true, G, M, N, n, EPI_ACC_F32, N, nullptr, 0, nullptr, 0, nullptr, 0,
                               slices));
      };
      // MLP half: y = x1 + g2 * (act w2^T). dact = (dy * g2) w2 never reaches memory: the epilogue turns it into du
      return wgrad(12, dy, D, c.act, F, g.G2) &&
             run(13, gemm(dy, false, g.w2g, true, g.du, n, F, D, EPI_SWIGLU_BWD, 2 * F, u, 2 * F)) &&
             run(14, gemm(g.du, false, b.w1, true, g.dh, n, D, 2 * F, EPI_STORE, D)) &&
             wgrad(15, g.du, 2 * F, c.h2, D, g.w1) &&
             run(16, aeris_modnorm_bwd(c.x1, g.dh, dy, v.scale2, v.shift2, b.wn2, g.dx1, dm + 4 * D, dm + 3 * D, g.n2, n, D,
                                       b.mode, b.eps, nullptr, b.stream)) &&
             // attention half: x1 = x + g1 * (o wo^T)
             wgrad(17, g.dx1, D, c.o, HD, g.Go) &&
             run(18, gemm(g.dx1, false, g.wog, true, g.d_o, n, HD, D, EPI_STORE, HD)) &&
             run(19, aeris_attn_bwd(c.qkv, 3 * HD, 0, HD, 2 * HD, c.o, g.d_o, HD, c.lse, g.delta, g.dqkv, 3 * HD, nw, b.L,
                                    b.heads, b.head_dim, b.scale, b.status, b.stream), 2) &&
             rope(b, run, 20, reinterpret_cast<bf16*>(g.dqkv), n, 1) &&
             run(21, gemm(g.dqkv, false, b.wqkv, true, g.dh, n, D, 3 * HD, EPI_STORE, D)) &&
             wgrad(22, g.dqkv, 3 * HD, c.h1, D, g.to_qkv) &&
             run(23, aeris_modnorm_bwd(x, g.dh, g.dx1, v.scale1, v.shift1, b.wn1, dx, dm + D, dm, g.n1, n, D, b.mode, b.eps,
                                       nullptr, b.stream));
    });
    if (!ok || !run(24, aeris_gate_finalize_pair(g.G2, b.w2, v.gate2, g.w2, dm + 5 * D, F, g.Go, b.wo, v.gate1, g.wo,
                                                 dm + 2 * D, HD, D, b.stream)))
      break;
  }
  return run.result();
}
