// Diffusion-side kernels around the transformer: everything between the image-layout fields on the device and the
// window-major token stream.
//   * embed_pack: TrigFlow noising with counter-based (Philox4x32-10) Gaussian noise, additive 2-D sinusoidal
//     position encoding, window partition by index arithmetic, and the split of the fp32 model input into bf16
//     (hi, lo) parts so that the K = 144 input projection runs on the tensor cores at fp32-level accuracy
//     (reference: src/aeris/parallelism/parallel_engine.py:21-33,673-678; src/aeris/models/parallel_swin.py:120-155,
//     383-386)
//   * trigflow_loss: weighted v-prediction loss and its gradient in one pass, the noise regenerated from the counter
//     (parallel_engine.py:990-997); the loss stays on the device
//   * sampler_update / noise_mix / affine_channels: Euler and Heun updates, churn and initial noise, and the
//     (un)standardisation + residual add of the rollout, all on the device (src/aeris/pp_generate.py:228-241,
//     298-333, which round-trips through host numpy)
// The noise of pixel (sample, Y, X), channel c depends only on the seed and on those global coordinates, so it does not
// change with the window-parallel or sequence-parallel layout of the run.
#include "common.cuh"
#include "api.h"

namespace aeris {

__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c.x), lo0 = 0xD2511F53u * c.x;
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c.z), lo1 = 0xCD9E8D57u * c.z;
    c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
    k.x += 0x9E3779B9u;
    k.y += 0xBB67AE85u;
  }
  return c;
}

__device__ __forceinline__ float u01(uint32_t r) { return (static_cast<float>(r >> 8) + 0.5f) * (1.0f / 16777216.0f); }

// Four independent N(0,1) draws for channels [4 * group, 4 * group + 4) of global pixel `pix`.
__device__ __forceinline__ float4 normal4(unsigned long long seed, unsigned long long pix, uint32_t group) {
  const uint4 r = philox4x32_10(make_uint4(static_cast<uint32_t>(pix), static_cast<uint32_t>(pix >> 32), group, 0x41455249u),
                                make_uint2(static_cast<uint32_t>(seed), static_cast<uint32_t>(seed >> 32)));
  const float r0 = sqrtf(-2.0f * logf(u01(r.x))), r1 = sqrtf(-2.0f * logf(u01(r.z)));
  float s0, c0, s1, c1;
  sincosf(6.283185307179586f * u01(r.y), &s0, &c0);
  sincosf(6.283185307179586f * u01(r.w), &s1, &c1);
  return make_float4(r0 * c0, r0 * s0, r1 * c1, r1 * s1);
}

struct Pixel {
  int b, y, x;
};
__device__ __forceinline__ int geom_rows_per_sample(const TokGeom& g) { return g.nwy_loc * g.nwx_loc * g.n_local; }
// Row of this rank's token stream (unshifted window layout, this rank's slice of every window's sequence) -> pixel
// of this rank's image block.
__device__ __forceinline__ Pixel row_to_pixel(const TokGeom& g, long long row) {
  const int rps = geom_rows_per_sample(g);
  Pixel p;
  // a 64-bit quotient takes as long as the rest of the row's addresses
  p.b = row >> 32 ? static_cast<int>(row / rps) : static_cast<int>(static_cast<uint32_t>(row) / static_cast<uint32_t>(rps));
  const int r = static_cast<int>(row - static_cast<long long>(p.b) * rps);
  const int w = r / g.n_local, tok = r - w * g.n_local;
  const int seq = g.sp_rank * g.n_local + tok;
  const int iy = seq / g.ws_x, ix = seq - iy * g.ws_x;
  const int wy = w / g.nwx_loc, wx = w - wy * g.nwx_loc;
  p.y = wy * g.ws_y + iy;
  p.x = wx * g.ws_x + ix;
  return p;
}
__device__ __forceinline__ unsigned long long global_pixel(const TokGeom& g, const Pixel& p) {
  return (static_cast<unsigned long long>(g.sample0 + p.b) * g.H + (g.y0 + p.y)) * g.W + (g.x0 + p.x);
}
__device__ __forceinline__ size_t block_pixel(const TokGeom& g, const Pixel& p) {
  return (static_cast<size_t>(p.b) * (g.nwy_loc * g.ws_y) + p.y) * (g.nwx_loc * g.ws_x) + p.x;
}

constexpr int EMBED_MAX_C = 256;
constexpr int EMBED_WARPS = 8;
constexpr int EMBED_LINE = (3 * EMBED_MAX_C + 2 + 7) / 8 * 8;      // columns of a packed row that can be other than zero

// Output row of a token: [hi(v) | lo(v) | hi(v) | 1 | 1 | 0...] of width KP (bf16), v the fp32 model input
// cat[x_t / sigma_d, cond] + ape. Multiplied by [hi(W) | hi(W) | lo(W) | hi(b) | lo(b) | 0...] this gives v W^T + b up to
// the dropped lo*lo term. Bound by instructions and their latency, not by its bytes, so:
//   * A warp takes `chunk` consecutive rows: a lane's addresses move by one pixel, and what has to be divided or multiplied
//     out is done once per row of a window.
//   * A lane takes W = 2 channels at a time where all counts are even and all tables start on 8 bytes, else one.
//   * The row is put together in shared memory, where its constant end stays from row to row, and leaves in 16-byte vectors
//     (`vec`; two-column words where `out` starts elsewhere): the parts of a channel are computed once.
// us, 70 + 74 channels, a row at a time with divisions per column / now (40 warps per SM, 48 registers): 64,800 rows
// 86 / 32, 14,400 22.6 / 9.6, 64,800 with noise 92 / 44; 259,200 rows of 69 + 71 channels 334 / 157.
// Its bytes take 16, 3.5, 16 and 63.
template <int W, bool NOISE>
__global__ void __launch_bounds__(EMBED_WARPS * 32, 5)
embed_pack_kernel(const float* __restrict__ x_img, const float* __restrict__ c_img, const float* __restrict__ cs,
                  TokGeom g, int Cx, int Cc, const float* __restrict__ ape_y, const float* __restrict__ ape_x,
                  int ape_ch, unsigned long long seed, float sd, __nv_bfloat16* __restrict__ out, int KP,
                  long long row0, long long rows, int chunk, int vec) {
  chain_point();
  constexpr int STEPS = EMBED_MAX_C / (32 * W);
  __shared__ __align__(16) __nv_bfloat16 lines[EMBED_WARPS][EMBED_LINE];
  __shared__ __align__(16) float zs[EMBED_WARPS][NOISE ? EMBED_MAX_C : 4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __nv_bfloat16* line = lines[warp];
  float* z = zs[warp];
  const int Cin = Cx + Cc;
  const float inv_sd = 1.0f / sd;
  for (int j = lane; j < EMBED_LINE; j += 32) line[j] = __float2bfloat16_rn(j >= 3 * Cin && j < 3 * Cin + 2 ? 1.f : 0.f);
  const long long first = (static_cast<long long>(blockIdx.x) * EMBED_WARPS + warp) * chunk;
  const int n = static_cast<int>(rows - first < chunk ? rows - first : chunk);
  Pixel p{};
  int tok = g.n_local, ix = 0;          // the first row is looked up
  float ct = 0.f, st = 0.f;
  // of the pixel, for channel 0 plus this lane's first: state, conditioning, position encoding of its row and column
  const float *xp = nullptr, *cp = nullptr, *ay = nullptr, *ax = nullptr;
  const int ape_c = ape_y ? 2 * ape_ch : 0;
  for (int k = 0; k < n; ++k) {
    const bool look_up = tok == g.n_local;
    if (look_up) {
      p = row_to_pixel(g, row0 + first + k);
      tok = static_cast<int>((row0 + first + k) % g.n_local);
      ix = (g.sp_rank * g.n_local + tok) % g.ws_x;
      ct = cs[2 * p.b];
      st = cs[2 * p.b + 1];
    }
    if (look_up || ix == 0) {
      const size_t bp = block_pixel(g, p);
      xp = x_img + bp * Cx + lane * W;
      cp = c_img + bp * Cc + lane * W - Cx;
      ay = ape_y + static_cast<size_t>(g.y0 + p.y) * ape_ch + lane * W;
      ax = ape_x + static_cast<size_t>(g.x0 + p.x) * ape_ch + lane * W - ape_ch;
    }
    if constexpr (NOISE) {
      const unsigned long long gp = global_pixel(g, p);
      for (int grp = lane; grp * 4 < Cx; grp += 32) *reinterpret_cast<float4*>(z + grp * 4) = normal4(seed, gp, grp);
    }
    __syncwarp();                       // the row before has left, this one's noise is there
#pragma unroll
    for (int i = 0; i < STEPS; ++i) {
      const int c = (lane + 32 * i) * W;
      if (c >= Cin) break;
      float f[W], a[W];
      auto load = [&](const float* at, float (&t)[W]) {
        if constexpr (W == 2) {
          const float2 u = *reinterpret_cast<const float2*>(at + 64 * i);
          t[0] = u.x;
          t[1] = u.y;
        } else {
          t[0] = at[32 * i];
        }
      };
      load(c < Cx ? xp : cp, f);
      if (c < ape_c) load(c < ape_ch ? ay : ax, a);
      if (c < Cx) {
#pragma unroll
        for (int h = 0; h < W; ++h) f[h] = NOISE ? (ct * f[h] + st * sd * z[c + h]) * inv_sd : ct * f[h] * inv_sd;
      }
      if (c < ape_c) {
#pragma unroll
        for (int h = 0; h < W; ++h) f[h] = __fadd_rn(f[h], a[h]);     // never one rounding with the product before it
      }
      if constexpr (W == 2) {
        const uint32_t hi = pack_bf16x2(f[0], f[1]);
        const float2 h = unpack_bf16x2(hi);
        *reinterpret_cast<uint32_t*>(line + c) = hi;
        *reinterpret_cast<uint32_t*>(line + Cin + c) = pack_bf16x2(f[0] - h.x, f[1] - h.y);
        *reinterpret_cast<uint32_t*>(line + 2 * Cin + c) = hi;
      } else {
        const __nv_bfloat16 hi = __float2bfloat16_rn(f[0]);
        line[c] = hi;
        line[Cin + c] = __float2bfloat16_rn(f[0] - __bfloat162float(hi));
        line[2 * Cin + c] = hi;
      }
    }
    __syncwarp();
    __nv_bfloat16* orow = out + static_cast<size_t>(first + k) * KP;
    if (vec) {
      for (int j = lane; j < KP / 8; j += 32)
        reinterpret_cast<uint4*>(orow)[j] =
            j < EMBED_LINE / 8 ? reinterpret_cast<const uint4*>(line)[j] : make_uint4(0u, 0u, 0u, 0u);
    } else {
      for (int j = lane; j < KP / 2; j += 32)
        reinterpret_cast<uint32_t*>(orow)[j] = j < EMBED_LINE / 2 ? reinterpret_cast<const uint32_t*>(line)[j] : 0u;
    }
    ++tok;
    ++p.x;
    xp += Cx;
    cp += Cc;
    ax += ape_ch;
    if (++ix == g.ws_x) {
      ix = 0;
      p.x -= g.ws_x;
      ++p.y;
    }
  }
}

// Loss and its gradient. pred: fp32 [rows, ldp] (network output F in token order); the target is
// v = cos(t) z sigma_d - sin(t) x. loss += sum_rows sum_c w_var[c] w_lat[Y] (sigma_d F - v)^2 * inv_rows;
// dpred (bf16 [rows, ldd], columns >= Cx zero) = d loss / d F * gscale.
__global__ void __launch_bounds__(EMBED_WARPS * 32)
trigflow_loss_kernel(const float* __restrict__ pred, int ldp, const float* __restrict__ x_img,
                     const float* __restrict__ cs, TokGeom g, int Cx, unsigned long long seed, float sd,
                     const float* __restrict__ w_var, const float* __restrict__ w_lat, float inv_rows, float gscale,
                     __nv_bfloat16* __restrict__ dpred, int ldd, double* __restrict__ loss, long long row0,
                     long long rows) {
  chain_point();
  __shared__ float part[EMBED_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float acc = 0.f;
  for (long long i = static_cast<long long>(blockIdx.x) * EMBED_WARPS + warp; i < rows;
       i += static_cast<long long>(gridDim.x) * EMBED_WARPS) {
    const Pixel p = row_to_pixel(g, row0 + i);
    const size_t bp = block_pixel(g, p);
    const unsigned long long gp = global_pixel(g, p);
    const float ct = cs[2 * p.b], st = cs[2 * p.b + 1];
    const float wl = w_lat ? w_lat[g.y0 + p.y] : 1.0f;
    const float* prow = pred + static_cast<size_t>(i) * ldp;
    for (int grp = lane; grp * 4 < ldd; grp += 32) {
      float d[4] = {0.f, 0.f, 0.f, 0.f};
      if (grp * 4 < Cx) {
        const float4 z = normal4(seed, gp, grp);
        const float zz[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int c = grp * 4 + k;
          if (c < Cx) {
            const float vt = ct * sd * zz[k] - st * x_img[bp * Cx + c];
            const float e = sd * prow[c] - vt;
            const float wgt = (w_var ? w_var[c] : 1.0f) * wl;
            acc += wgt * e * e;
            d[k] = 2.0f * sd * wgt * e * inv_rows * gscale;
          }
        }
      }
      if (dpred) {
        uint2 u;
        u.x = pack_bf16x2(d[0], d[1]);
        u.y = pack_bf16x2(d[2], d[3]);
        *reinterpret_cast<uint2*>(dpred + static_cast<size_t>(i) * ldd + grp * 4) = u;
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) part[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < EMBED_WARPS; ++w) s += part[w];
    atomicAdd(loss, static_cast<double>(s) * inv_rows);
  }
}

// x_out[pixel, c] = x_base[pixel, c] + ca * pa[row, c] + cb * pb[row, c]   (pa, pb in token order, x in image order)
__global__ void sampler_update_kernel(float* __restrict__ x_out, const float* __restrict__ x_base,
                                      const float* __restrict__ pa, const float* __restrict__ pb, int ldp, float ca,
                                      float cb, TokGeom g, int Cx, long long rows) {
  chain_point();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (long long i = static_cast<long long>(blockIdx.x) * nw + warp; i < rows;
       i += static_cast<long long>(gridDim.x) * nw) {
    const Pixel p = row_to_pixel(g, i);
    const size_t bp = block_pixel(g, p);
    for (int c = lane; c < Cx; c += 32) {
      float v = x_base[bp * Cx + c] + ca * pa[static_cast<size_t>(i) * ldp + c];
      if (pb) v += cb * pb[static_cast<size_t>(i) * ldp + c];
      x_out[bp * Cx + c] = v;
    }
  }
}

// x[pixel, c] = a * x[pixel, c] + b * z(pixel, c): initial noise (a = 0) and churn rotations of the sampler.
__global__ void noise_mix_kernel(float* __restrict__ x, float a, float b, unsigned long long seed, TokGeom g, int Cx,
                                 long long n_pix) {
  const int groups = (Cx + 3) / 4;
  const long long total = n_pix * groups;
  const int hb = g.nwy_loc * g.ws_y, wb = g.nwx_loc * g.ws_x;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long pix = i / groups;
    const int grp = static_cast<int>(i - pix * groups);
    Pixel p;
    p.b = static_cast<int>(pix / (static_cast<long long>(hb) * wb));
    const int rem = static_cast<int>(pix - static_cast<long long>(p.b) * hb * wb);
    p.y = rem / wb;
    p.x = rem - p.y * wb;
    const float4 z = normal4(seed, global_pixel(g, p), grp);
    const float zz[4] = {z.x, z.y, z.z, z.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = grp * 4 + k;
      if (c < Cx) {
        float* q = x + pix * Cx + c;
        *q = (a != 0.f ? a * *q : 0.f) + b * zz[k];
      }
    }
  }
}

// out[i] = in[i] * a[c] + b[c] (+ add[i]), c = i mod C: standardise, un-standardise, residual add of the rollout.
__global__ void affine_channels_kernel(float* __restrict__ out, const float* __restrict__ in,
                                       const float* __restrict__ a, const float* __restrict__ b,
                                       const float* __restrict__ add, long long n, int C) {
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int c = static_cast<int>(i % C);
    float v = in[i] * a[c] + b[c];
    if (add) v += add[i];
    out[i] = v;
  }
}

}  // namespace aeris

using namespace aeris;
extern int aeris_num_sms();

static inline int warp_grid(long long rows, int warps_per_cta) {
  long long b = (rows + warps_per_cta - 1) / warps_per_cta;
  const long long cap = static_cast<long long>(aeris_num_sms()) * 16;
  if (b > cap) b = cap;
  return static_cast<int>(b < 1 ? 1 : b);
}
static inline bool geom_ok(const TokGeom* g) {
  return g && g->B > 0 && g->nwy_loc > 0 && g->nwx_loc > 0 && g->ws_y > 0 && g->ws_x > 0 && g->n_local > 0 &&
         g->sp_rank >= 0 && (g->sp_rank + 1) * g->n_local <= g->ws_y * g->ws_x;
}

extern "C" int aeris_embed_pack(const float* x_img, const float* c_img, const float* cs, const TokGeom* g, int Cx,
                                int Cc, const float* ape_y, const float* ape_x, int ape_ch,
                                unsigned long long seed, float sd, int noise, void* out, int KP, long long row0,
                                long long rows, void* stream) {
  if (!geom_ok(g) || Cx <= 0 || Cc < 0 || Cx + Cc > EMBED_MAX_C || KP % 8 || KP < 3 * (Cx + Cc) + 2 || rows <= 0)
    return -1;
  if (row0 < 0 || row0 + rows > static_cast<long long>(g->B) * g->nwy_loc * g->nwx_loc * g->n_local) return -2;
  // 40 warps per SM, of consecutive rows each; two channels a lane where pairs of them are whole 8-byte words
  const long long warps = static_cast<long long>(aeris_num_sms()) * 40;
  const long long chunk = (rows + warps - 1) / warps, ctas = ((rows + chunk - 1) / chunk + EMBED_WARPS - 1) / EMBED_WARPS;
  if (chunk > 0x7fffffff) return -1;
  const uintptr_t at = reinterpret_cast<uintptr_t>(x_img) | reinterpret_cast<uintptr_t>(c_img) |
                       reinterpret_cast<uintptr_t>(ape_y) | reinterpret_cast<uintptr_t>(ape_x);
  const bool two = (Cx | Cc | ape_ch) % 2 == 0 && at % 8 == 0;
  auto kern = noise ? (two ? embed_pack_kernel<2, true> : embed_pack_kernel<1, true>)
                    : (two ? embed_pack_kernel<2, false> : embed_pack_kernel<1, false>);
  return launch_chained(kern, static_cast<unsigned>(ctas), EMBED_WARPS * 32, 0, reinterpret_cast<cudaStream_t>(stream),
                        x_img, c_img, cs, *g, Cx, Cc, ape_y, ape_x, ape_ch, seed, sd, reinterpret_cast<__nv_bfloat16*>(out),
                        KP, row0, rows, static_cast<int>(chunk), (reinterpret_cast<uintptr_t>(out) & 15) == 0);
}

extern "C" int aeris_trigflow_loss(const float* pred, int ldp, const float* x_img, const float* cs, const TokGeom* g,
                                   int Cx, unsigned long long seed, float sd, const float* w_var, const float* w_lat,
                                   float inv_rows, float gscale, void* dpred, int ldd, double* loss, long long row0,
                                   long long rows, void* stream) {
  if (!geom_ok(g) || Cx <= 0 || Cx > ldp || ldd % 4 || (dpred && Cx > ldd) || rows <= 0) return -1;
  if (row0 < 0 || row0 + rows > static_cast<long long>(g->B) * g->nwy_loc * g->nwx_loc * g->n_local) return -2;
  return launch_chained(trigflow_loss_kernel, warp_grid(rows, EMBED_WARPS), EMBED_WARPS * 32, 0,
                        reinterpret_cast<cudaStream_t>(stream), pred, ldp, x_img, cs, *g, Cx, seed, sd, w_var, w_lat,
                        inv_rows, gscale, reinterpret_cast<__nv_bfloat16*>(dpred), ldd, loss, row0, rows);
}

extern "C" int aeris_sampler_update(float* x_out, const float* x_base, const float* pa, const float* pb, int ldp,
                                    float ca, float cb, const TokGeom* g, int Cx, void* stream) {
  if (!geom_ok(g) || Cx <= 0 || Cx > ldp) return -1;
  const long long rows = static_cast<long long>(g->B) * g->nwy_loc * g->nwx_loc * g->n_local;
  return launch_chained(sampler_update_kernel, warp_grid(rows, 8), 256, 0, reinterpret_cast<cudaStream_t>(stream), x_out,
                        x_base, pa, pb, ldp, ca, cb, *g, Cx, rows);
}

extern "C" int aeris_noise_mix(float* x, float a, float b, unsigned long long seed, const TokGeom* g, int Cx,
                               void* stream) {
  if (!geom_ok(g) || Cx <= 0) return -1;
  const long long n_pix = static_cast<long long>(g->B) * g->nwy_loc * g->ws_y * g->nwx_loc * g->ws_x;
  const long long work = n_pix * ((Cx + 3) / 4);
  long long blocks = (work + 255) / 256;
  const long long cap = static_cast<long long>(aeris_num_sms()) * 16;
  if (blocks > cap) blocks = cap;
  noise_mix_kernel<<<static_cast<int>(blocks), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(x, a, b, seed, *g,
                                                                                                 Cx, n_pix);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

extern "C" int aeris_affine_channels(float* out, const float* in, const float* a, const float* b, const float* add,
                                     long long n, int C, void* stream) {
  if (n <= 0 || C <= 0) return -1;
  long long blocks = (n + 255) / 256;
  const long long cap = static_cast<long long>(aeris_num_sms()) * 16;
  if (blocks > cap) blocks = cap;
  affine_channels_kernel<<<static_cast<int>(blocks), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(out, in, a, b,
                                                                                                       add, n, C);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}
