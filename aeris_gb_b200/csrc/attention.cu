// Windowed multi-head attention for sm_100a: softmax(Q K^T * scale) V per (window, head), non-causal and unmasked,
// forward and backward, flash-style (no N x N matrix in memory), on tcgen05 tensor cores with TMEM accumulators.
//
// Reference semantics: src/aeris/models/parallel_swin.py:257-258 (F.scaled_dot_product_attention, is_causal=False)
// and src/aeris_wp_inference/model.py:289-309 (naive softmax(QK^T)V over each window's tokens).
//
// Data layout: tokens are window-major, rows [w*N, (w+1)*N) belong to window w; Q, K, V are column slices of a
// row-major [T, ld] bf16 tensor (the fused qkv projection output, columns ordered (q|k|v, head, d)).
//
// Roles in the kernels of this file: warp 0 = TMA producer, warp 1 = MMA issuer and TMEM owner, and warpgroups of math
// warps, one thread per tile row, that work straight out of TMEM. The forward kernel has one such group (warps 2..5 of 192
// threads). The backward kernels have two or three from warp 4 on (384 or 512 threads); warps 2 and 3 fetch the row
// statistics there. The forward kernel for windows of several query tiles (attention_fwd_pair.cuh) has its two softmax
// groups first, then a producer warp and one issuer warp per group.
#include "common.cuh"
#include "api.h"
#include "host.h"

namespace aeris {

constexpr int ATT_THREADS = 192;
constexpr int TILE = 128;

struct AttnFwdParams {
  __nv_bfloat16* O;
  int ldo;
  float* lse;  // [n_win * H * N], log2 domain: m + log2(l)
  int N, H, n_win;
  int d;         // head width, at most the kernel's HD (the tensor maps pad with zeros)
  float scale_log2;
  int* status;
  // Ulysses output push (all null / 0 when unused): row `grow` of window `win` belongs to rank grow / push_n_local and
  // is stored at row win * push_n_local + grow % push_n_local, column push_col0 + head * d of that rank's buffer.
  void* o_peers[8];
  int push_n_local, push_ld, push_col0;
};

// Byte offset of 16-byte vector `v` (0..7) of row `r` inside a [rows x 64] bf16 tile stored with the 128-byte swizzle.
__device__ __forceinline__ uint32_t swz128(int r, int v) { return r * 128 + (((v ^ (r & 7)) & 7) << 4); }

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Packed two-wide fp32 arithmetic (sm_100 f32x2 instructions): one issue slot per two scores.
__device__ __forceinline__ float mufu_exp2(float x) {   // not volatile: the scheduler may interleave it freely
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 2^x for a pair of exponents on the FMA pipe instead of the exp unit (which limits attention at head_dim 64):
// x = r + f with r = round(x), f in [-0.5, 0.5]; 2^f by a cubic (relative error 7.5e-5, far below bf16 resolution),
// 2^r by adding r to the exponent field. x is clamped at -125 so the exponent field cannot wrap; callers keep x <= 8.
__device__ __forceinline__ void poly_exp2_pair(uint64_t t2, float& p0, float& p1) {
  float t0, t1;
  f2_unpack(t2, t0, t1);
  t2 = f2_pack(fmaxf(t0, -125.f), fmaxf(t1, -125.f));
  const uint64_t magic = f2_pack(12582912.f, 12582912.f);     // 1.5 * 2^23: the sum's low mantissa bits hold round(x)
  const uint64_t tm = f2_add(t2, magic);
  const uint64_t f = f2_sub(t2, f2_sub(tm, magic));
  uint64_t q = f2_fma(f2_pack(0.0551716574f, 0.0551716574f), f, f2_pack(0.2426111251f, 0.2426111251f));
  q = f2_fma(q, f, f2_pack(0.6932609677f, 0.6932609677f));
  q = f2_fma(q, f, f2_pack(0.9999280572f, 0.9999280572f));
  float q0, q1, m0, m1;
  f2_unpack(q, q0, q1);
  f2_unpack(tm, m0, m1);
  p0 = __uint_as_float(__float_as_uint(m0) * 0x00800000u + __float_as_uint(q0));
  p1 = __uint_as_float(__float_as_uint(m1) * 0x00800000u + __float_as_uint(q1));
}

// Probabilities of one 64-score row segment (raw scores in v0 | v1) against the reference maximum m_ref: bf16 pairs
// into pk, their sum returned. POLY of every eight pairs take the polynomial path, the rest the exp unit, interleaved
// so that both pipes stay busy.
template <int POLY>
__device__ __forceinline__ float softmax_row64(const uint32_t (&v0)[32], const uint32_t (&v1)[32], float sl2,
                                               float m_ref, uint32_t (&pk)[32]) {
  const uint64_t sl = f2_pack(sl2, sl2), nm = f2_pack(-m_ref, -m_ref);
  uint64_t acc[4] = {0ull, 0ull, 0ull, 0ull};      // bit pattern of (0.f, 0.f)
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    const uint32_t a = (i < 16) ? v0[2 * i] : v1[2 * i - 32], b = (i < 16) ? v0[2 * i + 1] : v1[2 * i - 31];
    const uint64_t t = f2_fma(f2_pack(__uint_as_float(a), __uint_as_float(b)), sl, nm);
    float p0, p1;
    if ((i & 7) < POLY) {
      poly_exp2_pair(t, p0, p1);
    } else {
      float t0, t1;
      f2_unpack(t, t0, t1);
      p0 = mufu_exp2(t0);
      p1 = mufu_exp2(t1);
    }
    acc[i & 3] = f2_add(acc[i & 3], f2_pack(p0, p1));
    pk[i] = pack_bf16x2(p0, p1);
  }
  float s0, s1;
  f2_unpack(f2_add(f2_add(acc[0], acc[1]), f2_add(acc[2], acc[3])), s0, s1);
  return s0 + s1;
}

// -------------------------------------------------------------------------------------------------------- forward
// grid = (q_tiles, H, n_win). One CTA owns a 128-row Q tile and streams the window's K/V in 64-row tiles through a
// two-stage TMA ring. Per tile: S = Q K^T lands in TMEM, the four softmax warps (one thread per query row) read its 64
// scores once into registers and release the buffer at once, so the tensor core computes the next tile's scores under
// the exponentials; the bf16 probabilities go to shared memory as the A operand of P V, which ACCUMULATES in one TMEM
// buffer over all tiles. The running output is therefore never read back per tile: the exponentials use a reference
// maximum that is only raised (and the TMEM accumulator and row sum rescaled) when a row's maximum grows by more than
// 2^8, which bounds the probabilities by 256 and is exact after the final division by the row sum. The small footprint
// (64 KB shared memory, 128 TMEM columns, no register-resident output) lets three CTAs share an SM at head_dim 64.
constexpr int KVT = 64;
constexpr float RESCALE_LOG2 = 8.0f;

__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// acc[lane row, 0..cols) *= alpha in TMEM, eight columns at a time: it runs only when a row maximum jumps and must not add
// to the register pressure of the caller, whose 64 scores are live.
__device__ __forceinline__ void rescale_tmem_rows(uint32_t taddr, int cols, float alpha) {
#pragma unroll 1
  for (int c = 0; c < cols; c += 8) {
    uint32_t v[8];
    tmem_ld8(taddr + c, v);
    tmem_wait_ld();
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
    tmem_st8(taddr + c, v);
  }
  tmem_wait_st();
}

// Depth of the K and V rings of the forward kernel: at head_dim 64 three CTAs of 72 KB share an SM, at 128 two of 112 KB.
#ifdef AERIS_ATTN_TRACE
// Measurement build only: warp 2, lane 0 of CTA (0, 0, 0) stamps clock64 at the phase boundaries of every tile.
__device__ long long* g_attn_trace = nullptr;
#define ATTN_STAMP(slot) do { if (trace_on) g_attn_trace[(j) * 8 + (slot)] = clock64(); } while (0)
#else
#define ATTN_STAMP(slot) do { } while (0)
#endif

// Forward kernel modes. 0: probabilities through shared memory, three CTAs per SM at head_dim 64. 1: probabilities in
// tensor memory, over the score columns they came from (P V takes its A operand from TMEM). 2: as 1 with four lighter
// CTAs per SM. (A variant with two score buffers, which computes the scores of tile j + 1 under the softmax of tile j
// without the shared-memory round trip, fits only two CTAs per SM and measured no faster.)
template <int DCH, int MODE> struct AttnFwdRing {
  static constexpr int NSK = (DCH == 1 && MODE != 2) ? 3 : 2;
  static constexpr int NSV = 2;
  static constexpr int MIN_CTAS = (DCH == 2) ? 2 : (MODE == 2 ? 4 : 3);
};

// POLY < 0: scalar softmax arithmetic, every exponential on the exp unit; POLY >= 0: two-wide fp32 arithmetic with POLY of
// every eight score pairs exponentiated by the polynomial.
// PTMEM: the probabilities never touch shared memory. Each softmax thread writes its row of bf16 pairs back into the
// TMEM columns it has just read the scores from, and P V takes its A operand from tensor memory. An M128 x N64 x K16
// product with both operands in shared memory reads 6 KB for 32 cycles of math, more than the 128 B/cycle the shared
// memory delivers, so the kernel with P in shared memory (16 KB written and 16 KB read back per tile, on top of
// Q, K and V) is bound by shared-memory bandwidth rather than by the tensor or the exp unit.
template <int DCH, int POLY, int MODE>
__global__ void __launch_bounds__(ATT_THREADS, AttnFwdRing<DCH, MODE>::MIN_CTAS)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_v, const AttnFwdParams p) {
  constexpr int HD = 64 * DCH;
  constexpr int Q_BYTES = DCH * 16384;
  constexpr int T_BYTES = DCH * 8192;       // one K tile or one V tile (64 rows)
  // K and V travel in rings of their own: a K tile is free as soon as its Q K^T has completed, a whole softmax before
  // the V tile of the same step, so its successor is requested that much earlier and the load latency hides behind
  // the softmax of the tiles in between.
  constexpr bool PTMEM = MODE != 0;
  constexpr int NSK = AttnFwdRing<DCH, MODE>::NSK, NSV = AttnFwdRing<DCH, MODE>::NSV;
  constexpr int P_BYTES = PTMEM ? 0 : 16384;   // [128 x 64] bf16
  constexpr int TMEM_COLS = (DCH == 1) ? 128 : 256;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;
  uint8_t* sKr = sQ + Q_BYTES;
  uint8_t* sVr = sKr + NSK * T_BYTES;
  uint8_t* sP = sVr + NSV * T_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sP + P_BYTES);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;     // [NSK <= 4]
  uint64_t* k_empty = bars + 5;    // [NSK <= 4]
  uint64_t* v_full = bars + 9;     // [NSV <= 4]
  uint64_t* v_empty = bars + 13;   // [NSV <= 4]
  uint64_t* s_full = bars + 17;    // scores of tile j are in TMEM
  uint64_t* s_free = bars + 18;    // every softmax warp has read them into registers
  uint64_t* p_full = bars + 19;    // probabilities of tile j are in shared memory
  uint64_t* pv_done = bars + 20;   // P V of tile j has completed (P buffer reusable, accumulator up to date)
  static_assert(NSK <= 4 && NSV <= 4, "barrier slots");
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int qt = blockIdx.x, head = blockIdx.y, win = blockIdx.z;
  const int N = p.N;
  const int nfull = N / KVT, rem = N - nfull * KVT;
  const int nkv = nfull + (rem ? 1 : 0);
  const int n_last = rem ? ((rem + 15) & ~15) : KVT;  // MMA N of the last K/V tile

  if (threadIdx.x == 0) {
    int ab = (p.status && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
    if ((smem_u32(smem) & 1023u) != 0) {
      ab = 1;
      if (p.status) atomicCAS(p.status, 0, ERR_BOUNDS);
    }
    *s_abort = ab;
  }
  __syncthreads();
  if (*s_abort) return;

  if (threadIdx.x == 0) {
    prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v);
    mbar_init(q_full, 1);
    for (int i = 0; i < NSK; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); }
    for (int i = 0; i < NSV; ++i) { mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
    // only the softmax warps that own at least one real query row take part in the hand-shakes: a warp without rows
    // would run a tile ahead of the others and its arrivals would complete a phase that belongs to the slower warps
    const int n_valid_warps = min(4, (N - qt * TILE + 31) / 32);
    mbar_init(s_full, 1); mbar_init(s_free, n_valid_warps); mbar_init(p_full, n_valid_warps); mbar_init(pv_done, 1);
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tS = tmem_base;          // S : 64 columns
  const uint32_t tO = tmem_base + 64;     // O : HD columns, accumulated over all tiles

  if (warp == 0) {
    if (elect_one_sync()) {
      mbar_expect_tx(q_full, Q_BYTES);
#pragma unroll
      for (int c = 0; c < DCH; ++c)
        tma_load_4d(sQ + c * 16384, &tm_q, q_full, c * 64, head, qt * TILE, win);
      // K_i, then V_{i-1}: the order in which their slots come free (K_i after Q K^T of tile i - NSK, V_{i-1} after P V
      // of tile i - 1 - NSV, which completes later), so no wait holds up a load whose slot is already free
      for (int i = 0; i <= nkv; ++i) {
        if (i < nkv) {
          const int st = i % NSK;
          if (!mbar_wait(&k_empty[st], ((i / NSK) & 1) ^ 1, p.status, ERR_TIMEOUT_ATTN)) break;
          mbar_expect_tx(&k_full[st], T_BYTES);
#pragma unroll
          for (int c = 0; c < DCH; ++c)
            tma_load_4d(sKr + st * T_BYTES + c * 8192, &tm_k, &k_full[st], c * 64, head, i * KVT, win);
        }
        if (i >= 1) {
          const int j = i - 1, st = j % NSV;
          if (!mbar_wait(&v_empty[st], ((j / NSV) & 1) ^ 1, p.status, ERR_TIMEOUT_ATTN)) break;
          mbar_expect_tx(&v_full[st], T_BYTES);
#pragma unroll
          for (int c = 0; c < DCH; ++c)
            tma_load_4d(sVr + st * T_BYTES + c * 8192, &tm_v, &v_full[st], c * 64, head, j * KVT, win);
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one_sync()) {
      bool ok = mbar_wait(q_full, 0, p.status, ERR_TIMEOUT_ATTN);
      const uint32_t aQ = smem_u32(sQ), aP = smem_u32(sP), aKr = smem_u32(sKr), aVr = smem_u32(sVr);
      // S = Q K_j^T  (A = Q K-major, B = K K-major, reduction over d)
      auto issue_qk = [&](int j) -> bool {
        const int st = j % NSK;
        if (!mbar_wait(&k_full[st], (j / NSK) & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
        tc_fence_after();
        const int ncur = (j == nkv - 1) ? n_last : KVT;
        const uint32_t aK = aKr + st * T_BYTES;
        const uint32_t idesc_qk = make_idesc_bf16(TILE, ncur, 0, 0);
#pragma unroll
        for (int kk = 0; kk < 4 * DCH; ++kk) {
          const uint32_t qoff = (kk >> 2) * 16384 + (kk & 3) * 32;
          const uint32_t koff = (kk >> 2) * 8192 + (kk & 3) * 32;
          umma_ss(tS, make_smem_desc(aQ + qoff, 0, 1024), make_smem_desc(aK + koff, 0, 1024), idesc_qk, kk > 0);
        }
        tc_commit(s_full);
        tc_commit(&k_empty[st]);       // the K tile is free once these products have completed
        return true;
      };
      if (ok) ok = issue_qk(0);
      for (int j = 0; j < nkv && ok; ++j) {
        const int st = j % NSV;
        const int ncur = (j == nkv - 1) ? n_last : KVT;
        if constexpr (!PTMEM) {
          if (j + 1 < nkv) {     // the next tile's scores, as soon as this tile's have been read out of TMEM
            if (!mbar_wait(s_free, j & 1, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
            tc_fence_after();
            if (!issue_qk(j + 1)) { ok = false; break; }
          }
        }
        if (!mbar_wait(&v_full[st], (j / NSV) & 1, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
        if (!mbar_wait(p_full, j & 1, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
        tc_fence_after();
        // O += P_j V_j  (A = P K-major over kv, B = V MN-major: d contiguous, kv rows strided)
        const uint32_t aV = aVr + st * T_BYTES;
        const uint32_t idesc_pv = make_idesc_bf16(TILE, HD, 0, 1);
        for (int kk = 0; kk < ncur / 16; ++kk) {
          const uint32_t acc = (j > 0 || kk > 0) ? 1u : 0u;
          if constexpr (PTMEM)      // A = P in the score columns: 16 bf16 = 8 columns per K step
            umma_ts(tO, tS + kk * 8, make_smem_desc(aV + kk * 2048, 8192, 1024), idesc_pv, acc);
          else
            umma_ss(tO, make_smem_desc(aP + kk * 32, 0, 1024), make_smem_desc(aV + kk * 2048, 8192, 1024), idesc_pv, acc);
        }
        tc_commit(pv_done);
        tc_commit(&v_empty[st]);
        if constexpr (PTMEM) {
          // the tensor core executes in issue order: these scores overwrite P_j only after P_j V_j has consumed it
          if (j + 1 < nkv && !issue_qk(j + 1)) { ok = false; break; }
        }
      }
    }
  } else {
    const int q = warp & 3;
    const int row = q * 32 + lane;            // row inside the Q tile == TMEM lane
    const int grow = qt * TILE + row;         // row inside the window
    const bool warp_valid = (qt * TILE + q * 32) < N;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const float sl2 = p.scale_log2;
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    // Raises the reference maximum to m_new: rescales the TMEM accumulator (once P V of the previous tile is done) and l.
    auto rescale = [&](int j, float m_new, bool& waited) -> bool {
      if (j > 0) {
        if (!mbar_wait(pv_done, (j - 1) & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
        waited = true;
        tc_fence_after();
        const float alpha = fast_exp2(m_ref - m_new);
        rescale_tmem_rows(tO + lane_addr, HD, alpha);
        tc_fence_before();
        l *= alpha;
      }
      m_ref = m_new;
      return true;
    };
#ifdef AERIS_ATTN_TRACE
    const bool trace_on = g_attn_trace != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 &&
                          warp == 2 && lane == 0;
#endif
    for (int j = 0; j < nkv && ok && warp_valid; ++j) {
      const bool last = (j == nkv - 1);
      ATTN_STAMP(0);
      const uint32_t tSj = tS;
      if (!mbar_wait(s_full, j & 1, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
      tc_fence_after();
      ATTN_STAMP(1);
      bool waited = false;
      if (!last || rem == 0) {
        // full 64-column tile: one TMEM read, scores stay in registers, the TMEM buffer is released at once
        uint32_t v0[32], v1[32];
        if (warp_valid) {
          tmem_ld32(tSj + lane_addr, v0);
          tmem_ld32(tSj + lane_addr + 32, v1);
          tmem_wait_ld();
        }
        ATTN_STAMP(2);
        if constexpr (!PTMEM) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(s_free);
        }
        if (warp_valid) {
          // four independent chains of eight 3-input maxima instead of one chain of thirty-two
          float mxc[4];
#pragma unroll
          for (int c = 0; c < 4; ++c)
            mxc[c] = fmaxf(__uint_as_float(v0[c]), __uint_as_float(v1[c]));
#pragma unroll
          for (int i = 1; i < 8; ++i) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              mxc[c] = max3(mxc[c], __uint_as_float(v0[4 * i + c]), __uint_as_float(v1[4 * i + c]));
          }
          const float mx = fmaxf(max3(mxc[0], mxc[1], mxc[2]), mxc[3]);
          const float m_new = fmaxf(m_ref, mx * sl2);
          if (__any_sync(0xffffffffu, m_new - m_ref > RESCALE_LOG2)) {
            if (!rescale(j, m_new, waited)) { ok = false; break; }
          }
          ATTN_STAMP(3);
          uint32_t pk[32];
          if constexpr (POLY >= 0) {
            l += softmax_row64<POLY>(v0, v1, sl2, m_ref, pk);
          } else {
            float rs[4] = {0.f, 0.f, 0.f, 0.f};
  #pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float p0 = fast_exp2(fmaf(__uint_as_float(v0[2 * i]), sl2, -m_ref));
              const float p1 = fast_exp2(fmaf(__uint_as_float(v0[2 * i + 1]), sl2, -m_ref));
              rs[(2 * i) & 3] += p0; rs[(2 * i + 1) & 3] += p1;
              pk[i] = pack_bf16x2(p0, p1);
            }
  #pragma unroll
            for (int i = 0; i < 16; ++i) {
              const float p0 = fast_exp2(fmaf(__uint_as_float(v1[2 * i]), sl2, -m_ref));
              const float p1 = fast_exp2(fmaf(__uint_as_float(v1[2 * i + 1]), sl2, -m_ref));
              rs[(2 * i) & 3] += p0; rs[(2 * i + 1) & 3] += p1;
              pk[16 + i] = pack_bf16x2(p0, p1);
            }
            l += (rs[0] + rs[1]) + (rs[2] + rs[3]);
          }
          ATTN_STAMP(4);
          if constexpr (PTMEM) {
            // scores of tile j exist, so P V of tile j - 1 (issued before them) is done: the columns are this thread's
            tmem_st32(tSj + lane_addr, pk);
            tmem_wait_st();
          } else {
            if (j > 0 && !waited && !mbar_wait(pv_done, (j - 1) & 1, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
#pragma unroll
            for (int g = 0; g < 8; ++g)
              *reinterpret_cast<uint4*>(sP + swz128(row, g)) =
                  make_uint4(pk[4 * g], pk[4 * g + 1], pk[4 * g + 2], pk[4 * g + 3]);
          }
        }
      } else {
        // last, partial tile: n_last (multiple of 16) columns computed, `rem` of them valid; no tile follows
        if (warp_valid) {
          float mx = -INFINITY;
#pragma unroll 1
          for (int c = 0; c < n_last; c += 16) {
            uint32_t v[16];
            tmem_ld16(tSj + lane_addr + c, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (c + i < rem) mx = fmaxf(mx, __uint_as_float(v[i]));
          }
          const float m_new = fmaxf(m_ref, mx * sl2);
          if (__any_sync(0xffffffffu, m_new - m_ref > RESCALE_LOG2)) {
            if (!rescale(j, m_new, waited)) { ok = false; break; }
          }
          if constexpr (!PTMEM) {
            if (j > 0 && !waited && !mbar_wait(pv_done, (j - 1) & 1, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
          }
          float rs = 0.f;
#pragma unroll 1
          for (int c = 0; c < n_last; c += 16) {
            uint32_t v[16], pk[8];
            tmem_ld16(tSj + lane_addr + c, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              float p0 = fast_exp2(fmaf(__uint_as_float(v[2 * i]), sl2, -m_ref));
              float p1 = fast_exp2(fmaf(__uint_as_float(v[2 * i + 1]), sl2, -m_ref));
              if (c + 2 * i >= rem) p0 = 0.f;
              if (c + 2 * i + 1 >= rem) p1 = 0.f;
              rs += p0 + p1;
              pk[i] = pack_bf16x2(p0, p1);
            }
            if constexpr (PTMEM) {
              // 16 scores become 8 columns of bf16 pairs at column c / 2 <= c: only scores already consumed are overwritten
              tmem_st8(tSj + lane_addr + (c >> 1), pk);
            } else {
#pragma unroll
              for (int g = 0; g < 2; ++g)
                *reinterpret_cast<uint4*>(sP + swz128(row, (c >> 3) + g)) =
                    make_uint4(pk[4 * g], pk[4 * g + 1], pk[4 * g + 2], pk[4 * g + 3]);
            }
          }
          if constexpr (PTMEM) tmem_wait_st();
          l += rs;
        }
        if constexpr (!PTMEM) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(s_free);
        }
      }
      ATTN_STAMP(5);
      if constexpr (!PTMEM) fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);
      ATTN_STAMP(6);
    }
    if (ok && warp_valid && mbar_wait(pv_done, (nkv - 1) & 1, p.status, ERR_TIMEOUT_ATTN)) {
      tc_fence_after();
      {
        const float inv = 1.f / l;
        const size_t trow = static_cast<size_t>(win) * N + grow;
        __nv_bfloat16* dst = (p.O && grow < N) ? p.O + trow * p.ldo + head * p.d : nullptr;
        __nv_bfloat16* pdst = nullptr;
        if (p.push_n_local > 0 && grow < N) {
          const int owner = grow / p.push_n_local;
          pdst = reinterpret_cast<__nv_bfloat16*>(p.o_peers[owner]) +
                 (static_cast<size_t>(win) * p.push_n_local + (grow - owner * p.push_n_local)) * p.push_ld +
                 p.push_col0 + head * p.d;
        }
#pragma unroll
        for (int c = 0; c < HD; c += 32) {
          if (c >= p.d) break;
          uint32_t v[32];
          tmem_ld32(tO + lane_addr + c, v);
          tmem_wait_ld();
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint4 u;
            u.x = pack_bf16x2(__uint_as_float(v[8 * g]) * inv, __uint_as_float(v[8 * g + 1]) * inv);
            u.y = pack_bf16x2(__uint_as_float(v[8 * g + 2]) * inv, __uint_as_float(v[8 * g + 3]) * inv);
            u.z = pack_bf16x2(__uint_as_float(v[8 * g + 4]) * inv, __uint_as_float(v[8 * g + 5]) * inv);
            u.w = pack_bf16x2(__uint_as_float(v[8 * g + 6]) * inv, __uint_as_float(v[8 * g + 7]) * inv);
            const bool live = c + 8 * g < p.d;
            if (dst && live) *reinterpret_cast<uint4*>(dst + c + 8 * g) = u;
            if (pdst && live) *reinterpret_cast<uint4*>(pdst + c + 8 * g) = u;
          }
        }
        if (p.lse && grow < N) p.lse[(static_cast<size_t>(win) * p.H + head) * N + grow] = m_ref + log2f(l);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

static int g_fwd_smem_pad = 0;   // extra dynamic shared memory per CTA: lowers the number of CTAs per SM (measurements)

template <int DCH, int POLY, int MODE>
static int launch_attn_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                           const AttnFwdParams& p, cudaStream_t stream) {
  constexpr int SMEM = DCH * 16384 + (AttnFwdRing<DCH, MODE>::NSK + AttnFwdRing<DCH, MODE>::NSV) * DCH * 8192 +
                       (MODE != 0 ? 0 : 16384) + 256;
  static int configured = -1;
  auto kern = attn_fwd_kernel<DCH, POLY, MODE>;
  const int smem = SMEM + g_fwd_smem_pad;
  if (configured != smem) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return -20;
    configured = smem;
  }
  dim3 grid((p.N + TILE - 1) / TILE, p.H, p.n_win);
  kern<<<grid, ATT_THREADS, smem, stream>>>(tq, tk, tv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}


}  // namespace aeris

#include "attention_fwd_pair.cuh"

namespace aeris {

// -------------------------------------------------------------------------------------------------------- backward
// Two kernels, neither needs atomics:
//   attn_bwd_dq : items of one 128-row Q tile, K/V streamed in 64-row tiles.  S = Q K^T, dP = dO V^T,
//                 dS = P * (dP - delta), dQ = scale * sum dS K.   Also writes delta = rowsum(dO * O).
//   attn_bwd_dkv: items of one 128-row K/V tile, Q/dO streamed in 64-row tiles. S^T = K Q^T, dP^T = V dO^T,
//                 dV += P^T dO, dK = scale * sum dS^T Q.
// What bounds them is the chain MMA -> commit -> TMEM load -> exponentials -> hand-over -> MMA: every link costs 200-300
// cycles of latency, so one tile in flight leaves the tensor core idle most of the time. Both kernels therefore run
// one persistent CTA per SM with NWG warpgroups of math warps, each with score buffers of its own in tensor memory and
// every NWG-th tile of the stream, so NWG chains are always in flight; the chains run on across work items (operands of
// the next item are prefetched, its first scores are computed under the epilogue of the current one). P and dS go
// back into the tensor memory columns they came from and are the A operand of the accumulating products from there:
// no shared-memory round trip, and the B operand is all that those products read from shared memory.
// Both kernels together, before (two 32-column halves in flight per CTA, P and dS through shared memory) and now:
// 72 windows x 900 tokens, 24 heads x 64: 2.61 -> 1.72 ms; 12 heads x 128: 2.67 -> 1.49 ms; 16 windows x 3600 tokens,
// 12 heads x 128: 7.05 -> 3.80 ms (12 launches each from an idle clock; 1.91, 1.69 and 4.35 ms held for 0.6 s, at
// 1740, 1725 and 1665 MHz under the power cap).
struct AttnBwdParams {
  const __nv_bfloat16* O;   // forward output, [T, ldo]
  const __nv_bfloat16* dO;  // [T, ldo]
  int ldo;
  const float* lse;         // [n_win*H*N] log2 domain
  float* delta;             // [n_win*H*N]
  __nv_bfloat16* dQKV;      // [T, ldg] gradient of the fused qkv tensor
  int ldg;
  int N, H, n_win;
  int d;         // head width, at most the kernel's HD (the tensor maps pad with zeros)
  int q_col0, k_col0, v_col0;
  float scale_log2, scale;
  int* status;
  // Ulysses gradient push (null / 0 when unused): the gradient row of token `grow` goes to rank grow / push_n_local,
  // row win * push_n_local + grow % push_n_local, column section * push_sec_w + push_col0 + head * d.
  void* dq_peers[8];
  int push_n_local, push_ld, push_sec_w, push_col0;
};
constexpr int BT = 64;      // rows of a streamed tile

__device__ __forceinline__ __nv_bfloat16* bwd_dst(const AttnBwdParams& p, int win, int grow, int head, int section,
                                                  int local_col0) {
  if (p.push_n_local > 0) {
    const int owner = grow / p.push_n_local;
    return reinterpret_cast<__nv_bfloat16*>(p.dq_peers[owner]) +
           (static_cast<size_t>(win) * p.push_n_local + (grow - owner * p.push_n_local)) * p.push_ld +
           section * p.push_sec_w + p.push_col0 + head * p.d;
  }
  return p.dQKV + (static_cast<size_t>(win) * p.N + grow) * p.ldg + local_col0 + head * p.d;
}

// Chains, ring depth and copies of the item's own operands per head width; the shared memory of one CTA per SM (227 KB)
// and its 512 TMEM columns set them: NWG * 128 score columns + the accumulators (dQ: HD, dK and dV: 2 HD).
// The ring holds 2 * NWG tiles. That is also what makes `next_full` sound, the one barrier per chain and round that the
// MMA thread waits on: it completes when the four math warps have handed over tile t AND the loads of tile t + NWG have
// landed. The producer may arm it for tile t + NWG only when the previous round is complete, which the slot it waits
// for (freed by the products of tile t - NWG) implies. One wait, one fence and two commits per tile matter because each
// costs the MMA thread 60-200 cycles: with separate barriers for the operands that thread was the bottleneck.
template <int DCH> struct BwdRing {
  static constexpr int NWG = (DCH == 1) ? 3 : 2;
  static constexpr int NST = 2 * NWG;
  static constexpr int NB = (DCH == 1) ? 2 : 1;         // buffers for the item's own 128-row operands
  static constexpr int ITEM_BYTES = 2 * DCH * 16384, STAGE = 2 * DCH * 8192;
  static constexpr int STAT = 4 * TILE > NST * 2 * BT ? 4 * TILE : NST * 2 * BT;
  static constexpr bool STAGED = DCH == 2;              // gradient rows leave through shared memory, see BwdOut
  static constexpr int OUT_BYTES = STAGED ? 2 * TILE * 64 : 0;  // two buffers of 32 columns, per warpgroup
  static constexpr int SMEM = NB * ITEM_BYTES + NST * STAGE + NWG * OUT_BYTES + STAT * 4 + 512;
  static constexpr int THREADS = 128 + 128 * NWG;
};
static_assert(BwdRing<1>::SMEM <= 227 * 1024 && BwdRing<2>::SMEM <= 227 * 1024, "shared memory");

// Asynchronous 4-byte copy (`bytes` = 0: zero fill), and this lane's arrival on a barrier once its copies have landed.
__device__ __forceinline__ void cp_async4(float* smem_dst, const float* src, uint32_t bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(smem_dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Gradient rows on their way out: a warp turns 32 accumulator columns of its 32 rows into bf16 in shared memory, one lane
// hands them to the TMA unit as a tiled store. The accumulator is free once it has been read; written by the threads
// themselves (one row each, 32 rows with every 16-byte store instruction) it kept the next item's products waiting. Rows
// past the window's end and columns past the head's width are clipped by the tensor map. No warp waits for another one's
// rows. Both kernels, ms, direct stores / now, in turn, 12 heads x 128: 400 x 128 tokens 0.548 / 0.456, 200 x 225 0.631 /
// 0.535, 72 x 900 1.73 / 1.61, 16 x 3600 4.50 / 4.31; with one buffer a warp 0.527, 0.602, 1.59 and 4.35. At 64, with a
// third of the columns per warpgroup, staging (of a warpgroup's 128 rows at a time) cost more than it saved (24 x 64, 200 x
// 225: 0.650 -> 0.704, 72 x 900 1.91 -> 1.92): direct stores there.
struct BwdOut {
  uint8_t* stage;           // this warp's two: 32 rows of 64 bytes, the vectors of 16 swizzled as the tensor map has it
  int lane, first_row;      // of this warp inside the tile
  int n = 0;                // groups of columns so far

  // `read`: called once the columns are out of tensor memory
  template <typename F>
  __device__ __forceinline__ void put(uint32_t taddr, float f, const CUtensorMap* m, int col, int head, int tile_row,
                                      int win, int N, F&& read) {
    uint32_t v[32];
    tmem_ld32(taddr, v);
    tmem_wait_ld();
    read();
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
    __syncwarp();
    uint8_t* buf = stage + (n++ & 1) * 2048;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      uint32_t o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
        o[i] = pack_bf16x2(__uint_as_float(v[8 * g + 2 * i]) * f, __uint_as_float(v[8 * g + 2 * i + 1]) * f);
      *reinterpret_cast<uint4*>(buf + lane * 64 + ((g ^ ((lane >> 1) & 3)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      if (tile_row + first_row < N)
        tma_store_4d(m, buf, col, head, tile_row + first_row, win);
      else                  // no rows: an empty group, so that the buffers still come free in turn
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
    __syncwarp();           // the warp goes on as one: the next step reads tensor memory
  }
  // before this warp leaves: its copies have been performed
  __device__ __forceinline__ void drain() const {
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
};

// Position of a role in the CTA's stream of tiles: item `it` (of this CTA), tile `j` of the item, running number `g`.
struct TileIter {
  int it = 0, j = 0, g = 0;
  __device__ __forceinline__ void next(int n_tiles) {
    ++g;
    if (++j == n_tiles) { j = 0; ++it; }
  }
};
struct BwdItem {
  int tile, head, win;
};
// Items of one (window, head) are neighbours, so the CTAs at work share their streamed operands in L2.
__device__ __forceinline__ BwdItem bwd_item(int it, int n_row_tiles, int H) {
  const int idx = blockIdx.x + it * gridDim.x;
  const int wh = idx / n_row_tiles;
  BwdItem b;
  b.tile = idx - wh * n_row_tiles;
  b.win = wh / H;
  b.head = wh - b.win * H;
  return b;
}

template <int DCH>
__global__ void __launch_bounds__(128 + 128 * BwdRing<DCH>::NWG, 1)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                   const __grid_constant__ CUtensorMap tm_dq, const AttnBwdParams p, const int n_items_total) {
  using R = BwdRing<DCH>;
  constexpr int HD = 64 * DCH;
  constexpr int QB = DCH * 16384;       // Q tile, dO tile (128 rows)
  constexpr int KB = DCH * 8192;        // K tile, V tile (64 rows)
  constexpr int NWG = R::NWG, NST = R::NST, NB = R::NB;
  static_assert(NWG * 128 + HD <= 512, "TMEM columns");
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;                   // [NB] items: Q | dO
  uint8_t* sKV = sQ + NB * R::ITEM_BYTES;                    // [NST] K | V
  uint8_t* sOut = sKV + NST * R::STAGE;                      // [NWG]
  float* s_stat = reinterpret_cast<float*>(sOut + NWG * R::OUT_BYTES);   // [2] items: lse [128] | delta [128]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_stat + R::STAT);
  uint64_t* q_full = bars;              // [NB <= 2]
  uint64_t* q_empty = bars + 2;         // [NB]
  uint64_t* first_full = bars + 4;      // [NWG <= 3] K and V of the first tile of each chain
  uint64_t* next_full = bars + 7;       // [NWG] dS of the chain's tile is in TMEM, K and V of its next tile have landed
  uint64_t* kv_empty = bars + 10;       // [NST <= 6]
  uint64_t* sp_full = bars + 16;        // [NWG] scores and dP of a tile are in the chain's TMEM columns
  uint64_t* acc_full = bars + 19;
  uint64_t* acc_empty = bars + 20;
  uint64_t* stat_full = bars + 21;      // [2]
  uint64_t* stat_empty = bars + 23;     // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 25);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int N = p.N;
  const int nfull = N / BT, rem = N - nfull * BT;
  const int nkv = nfull + (rem ? 1 : 0);
  const int n_last = rem ? ((rem + 15) & ~15) : BT;
  const int row_tiles = (N + TILE - 1) / TILE;
  const int n_ctas = static_cast<int>(gridDim.x);
  const int n_items = (n_items_total - static_cast<int>(blockIdx.x) + n_ctas - 1) / n_ctas;

  if (threadIdx.x == 0) {
    int ab = (p.status && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
    if ((smem_u32(smem) & 1023u) != 0) { ab = 1; if (p.status) atomicCAS(p.status, 0, ERR_BOUNDS); }
    *s_abort = ab;
  }
  __syncthreads();
  if (*s_abort) return;
  if (threadIdx.x == 0) {
    prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v); prefetch_tmap(&tm_do);
    for (int i = 0; i < 2; ++i) { mbar_init(&stat_full[i], 2); mbar_init(&stat_empty[i], 4 * NWG); }
    for (int i = 0; i < NB; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
    for (int i = 0; i < NST; ++i) mbar_init(&kv_empty[i], 1);
    for (int i = 0; i < NWG; ++i) {
      mbar_init(&first_full[i], 1);
      mbar_init(&next_full[i], 4 + 1);
      mbar_init(&sp_full[i], 1);
    }
    mbar_init(acc_full, 1); mbar_init(acc_empty, 4 * NWG);
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tdQ = tmem_base + NWG * 128;      // chain w: S at w * 128, dP at w * 128 + 64

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one_sync()) {
      auto load_item = [&](int it) -> bool {
        const int b = it % NB;
        if (!mbar_wait(&q_empty[b], ((it / NB) & 1) ^ 1, p.status, ERR_TIMEOUT_ATTN)) return false;
        const BwdItem w = bwd_item(it, row_tiles, p.H);
        mbar_expect_tx(&q_full[b], R::ITEM_BYTES);
        uint8_t* d = sQ + b * R::ITEM_BYTES;
#pragma unroll
        for (int c = 0; c < DCH; ++c) {
          tma_load_4d(d + c * 16384, &tm_q, &q_full[b], c * 64, w.head, w.tile * TILE, w.win);
          tma_load_4d(d + QB + c * 16384, &tm_do, &q_full[b], c * 64, w.head, w.tile * TILE, w.win);
        }
        return true;
      };
      bool ok = load_item(0);
      int st = 0, t = 0;
      uint32_t ph = 1;
      // where an item's own operands are requested: with two buffers those of the next item early in this one, with one
      // buffer those of this item behind its first tiles (they have to wait for the last scores of the item before)
      const int j_item = min(NB == 2 ? 2 : NWG - 1, nkv - 1);
      for (int it = 0; it < n_items && ok; ++it) {
        const BwdItem w = bwd_item(it, row_tiles, p.H);
        for (int j = 0; j < nkv; ++j, ++t) {
          if (!mbar_wait(&kv_empty[st], ph, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
          uint64_t* bar = t < NWG ? &first_full[t] : &next_full[t % NWG];
          uint8_t* d = sKV + st * R::STAGE;
          mbar_expect_tx(bar, R::STAGE);
#pragma unroll
          for (int c = 0; c < DCH; ++c) {
            tma_load_4d(d + c * 8192, &tm_k, bar, c * 64, w.head, j * BT, w.win);
            tma_load_4d(d + KB + c * 8192, &tm_v, bar, c * 64, w.head, j * BT, w.win);
          }
          if (++st == NST) { st = 0; ph ^= 1; }
          if (j == j_item) {
            if (NB == 2 && it + 1 < n_items && !load_item(it + 1)) { ok = false; break; }
            if (NB == 1 && it > 0 && !load_item(it)) { ok = false; break; }
          }
        }
      }
      // the last tile of each chain has no successor: its round completes without loads
      for (int e = t + NWG; t < e && ok; ++t) {
        if (!mbar_wait(&kv_empty[st], ph, p.status, ERR_TIMEOUT_ATTN)) break;
        if (t >= NWG) mbar_arrive(&next_full[t % NWG]);
        if (++st == NST) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one_sync()) {
      const uint32_t aI = smem_u32(sQ), aS = smem_u32(sKV);
      const int total = n_items * nkv;
      TileIter s;                       // next tile whose scores are issued
      int s_w = 0, s_st = 0;
      // S = Q K_j^T and dP = dO V_j^T of tile s
      auto issue_sp = [&]() -> bool {
        const int b = s.it % NB;
        if (s.j == 0) {
          if (!mbar_wait(&q_full[b], (s.it / NB) & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
          tc_fence_after();
        }
        const bool last = s.j == nkv - 1;
        const uint32_t idesc = make_idesc_bf16(TILE, last ? n_last : BT, 0, 0);
        const uint32_t tS = tmem_base + s_w * 128;
        const uint64_t d0 = make_smem_desc(aI + b * R::ITEM_BYTES, 0, 1024), d1 = d0 + QB / 16;
        const uint64_t d2 = make_smem_desc(aS + s_st * R::STAGE, 0, 1024), d3 = d2 + KB / 16;
#pragma unroll
        for (int kk = 0; kk < 4 * DCH; ++kk)
          umma_ss(tS, d0 + ((kk >> 2) * 16384 + (kk & 3) * 32) / 16, d2 + ((kk >> 2) * 8192 + (kk & 3) * 32) / 16, idesc,
                  kk > 0);
#pragma unroll
        for (int kk = 0; kk < 4 * DCH; ++kk)
          umma_ss(tS + 64, d1 + ((kk >> 2) * 16384 + (kk & 3) * 32) / 16, d3 + ((kk >> 2) * 8192 + (kk & 3) * 32) / 16,
                  idesc, kk > 0);
        tc_commit(&sp_full[s_w]);
        if (last) tc_commit(&q_empty[b]);
        if (++s_w == NWG) s_w = 0;
        if (++s_st == NST) s_st = 0;
        s.next(nkv);
        return true;
      };
      bool ok = true;
      for (int i = 0; i < NWG && i < total && ok; ++i) {
        ok = mbar_wait(&first_full[i], 0, p.status, ERR_TIMEOUT_ATTN);
        tc_fence_after();
        if (ok) ok = issue_sp();
      }
      int w = 0, st = 0;
      uint32_t ph = 0;
      TileIter a;
      constexpr uint32_t idesc_acc = make_idesc_bf16(TILE, HD, 0, 1);
      while (ok && a.g < total) {
        if (!mbar_wait(&next_full[w], ph, p.status, ERR_TIMEOUT_ATTN)) break;
        if (a.j == 0 && a.it > 0 && !mbar_wait(acc_empty, (a.it - 1) & 1, p.status, ERR_TIMEOUT_ATTN)) break;
        tc_fence_after();
        const bool last = a.j == nkv - 1;
        const uint32_t acc0 = a.j > 0 ? 1u : 0u;
        const uint32_t tA = tmem_base + w * 128;
        // dQ += dS_j K_j : A = dS (TMEM, 16 kv columns = 8 words per K step), B = K MN-major (d contiguous)
        const uint64_t dk = make_smem_desc(aS + st * R::STAGE, 8192, 1024);
        if (!last || rem == 0) {
#pragma unroll
          for (int kk = 0; kk < BT / 16; ++kk) umma_ts(tdQ, tA + kk * 8, dk + kk * 128, idesc_acc, kk ? 1u : acc0);
        } else {
          for (int kk = 0; kk < n_last / 16; ++kk) umma_ts(tdQ, tA + kk * 8, dk + kk * 128, idesc_acc, kk ? 1u : acc0);
        }
        tc_commit(&kv_empty[st]);
        if (last) tc_commit(acc_full);
        // the tensor core executes in issue order: these scores overwrite the A operand above only after it was read
        if (s.g < total && !issue_sp()) break;
        if (++w == NWG) { w = 0; ph ^= 1; }
        if (++st == NST) st = 0;
        a.next(nkv);
      }
    }
  } else if (warp < 4) {
    // ------------------------------------------------------------ lse and delta of the rows of the coming items (two warps)
    constexpr int LPR = HD / 8, RPW = 32 / LPR;      // lanes per row, rows per warp and load
    constexpr int UN = 8;                            // loads in flight: an item must not wait for its statistics
    const int sub = lane % LPR, r0 = lane / LPR, half = (warp - 2) * (TILE / 2);
    for (int it = 0; it < n_items; ++it) {
      const int b = it & 1;
      if (!mbar_wait(&stat_empty[b], ((it >> 1) & 1) ^ 1, p.status, ERR_TIMEOUT_ATTN)) break;
      const BwdItem w = bwd_item(it, row_tiles, p.H);
      float* st = s_stat + b * 2 * TILE;
      const size_t sbase = (static_cast<size_t>(w.win) * p.H + w.head) * N + w.tile * TILE;
      const size_t obase = (static_cast<size_t>(w.win) * N + w.tile * TILE) * p.ldo + w.head * p.d + sub * 8;
      const int live = N - w.tile * TILE;            // rows of this tile inside the window
      float lse[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int row = half + u * 32 + lane;
        lse[u] = (row < live) ? p.lse[sbase + row] : 0.f;
      }
#pragma unroll 1
      for (int r = half; r < half + TILE / 2; r += RPW * UN) {
        uint4 a[UN], g[UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
          const int row = r + u * RPW + r0;
          a[u] = g[u] = make_uint4(0u, 0u, 0u, 0u);
          if (row < live && sub * 8 < p.d) {
            a[u] = *reinterpret_cast<const uint4*>(p.O + obase + static_cast<size_t>(row) * p.ldo);
            g[u] = *reinterpret_cast<const uint4*>(p.dO + obase + static_cast<size_t>(row) * p.ldo);
          }
        }
#pragma unroll
        for (int u = 0; u < UN; ++u) {
          const uint32_t aw[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, gw[4] = {g[u].x, g[u].y, g[u].z, g[u].w};
          float d = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 x = unpack_bf16x2(aw[i]), y = unpack_bf16x2(gw[i]);
            d = fmaf(x.x, y.x, d);
            d = fmaf(x.y, y.y, d);
          }
#pragma unroll
          for (int o = LPR / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
          const int row = r + u * RPW + r0;
          if (sub == 0) {
            st[TILE + row] = d;
            if (row < live) p.delta[sbase + row] = d;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) st[half + u * 32 + lane] = lse[u];
      __syncwarp();
      if (lane == 0) mbar_arrive(&stat_full[b]);
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------ math: one thread = one Q row, every NWG-th tile
    const int wg = (warp >> 2) - 1, q = warp & 3;
    const int row = q * 32 + lane;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t tS = tmem_base + lane_addr + wg * 128, tdP = tS + 64;
    const uint64_t sl = f2_pack(p.scale_log2, p.scale_log2);
    const float sc = p.scale;
    uint32_t ph = 0;
    int j = wg;                       // first tile of this warpgroup in the item at hand
    bool ok = true;
    BwdOut out{sOut + wg * R::OUT_BYTES + q * 4096, lane, q * 32};
    // Gradient rows of item `it` from TMEM to memory. Runs after this warpgroup's first tile of the NEXT item, so that the
    // wait for the last products of `it` is spent on that tile.
    auto epilogue = [&](int it) -> bool {
      if (!mbar_wait(acc_full, it & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
      tc_fence_after();
      const BwdItem w = bwd_item(it, row_tiles, p.H);
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty);
      };
      if (R::STAGED && p.push_n_local == 0) {
        int mine = 0;                   // this warpgroup's groups of 32 columns
        for (int c = wg * 32; c < p.d; c += 32 * NWG) ++mine;
        if (mine == 0) release();
        for (int c = wg * 32; c < p.d; c += 32 * NWG)
          out.put(tdQ + lane_addr + c, sc, &tm_dq, c, w.head, w.tile * TILE, w.win, N,
                  [&] { if (--mine == 0) release(); });
        return true;
      }
      const int grow = w.tile * TILE + row;
      const bool row_ok = grow < N;
      __nv_bfloat16* dst = bwd_dst(p, w.win, row_ok ? grow : 0, w.head, 0, p.q_col0);
#pragma unroll
      for (int c = 0; c < HD; c += 32) {
        if ((c / 32) % NWG != wg || c >= p.d) continue;
        uint32_t v[32];
        tmem_ld32(tdQ + lane_addr + c, v);
        tmem_wait_ld();
        if (row_ok) {
#pragma unroll
          for (int gq = 0; gq < 4; ++gq) {
            uint32_t o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              o[i] = pack_bf16x2(__uint_as_float(v[8 * gq + 2 * i]) * sc, __uint_as_float(v[8 * gq + 2 * i + 1]) * sc);
            if (c + gq * 8 < p.d) *reinterpret_cast<uint4*>(dst + c + gq * 8) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);
      return true;
    };
    for (int it = 0; it < n_items && ok; ++it) {
      bool pending = it > 0;
      const int b = it & 1;
      if (!mbar_wait(&stat_full[b], (it >> 1) & 1, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
      const float nlse = -s_stat[b * 2 * TILE + row], ndelta = -s_stat[b * 2 * TILE + TILE + row];
      __syncwarp();
      if (lane == 0) mbar_arrive(&stat_empty[b]);
      const uint64_t nl = f2_pack(nlse, nlse), nd = f2_pack(ndelta, ndelta);
      for (; j < nkv; j += NWG, ph ^= 1) {
        if (!mbar_wait(&sp_full[wg], ph, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
        tc_fence_after();
        if (j < nfull) {
#pragma unroll
          for (int c = 0; c < 64; c += 32) {
            uint32_t sv[32], dv[32], pk[16];
            tmem_ld32(tS + c, sv);
            tmem_ld32(tdP + c, dv);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              float t0, t1;
              f2_unpack(f2_fma(f2_pack(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), sl, nl), t0, t1);
              const uint64_t pr = f2_pack(mufu_exp2(t0), mufu_exp2(t1));
              const uint64_t df = f2_add(f2_pack(__uint_as_float(dv[2 * i]), __uint_as_float(dv[2 * i + 1])), nd);
              pk[i] = f2_to_bf16x2(f2_mul(pr, df));
            }
            // 32 scores become 16 words at column c / 2 <= c: only scores that were read are overwritten
            tmem_st16(tS + (c >> 1), pk);
          }
        } else {
          // columns past the window's end: their K rows are zeros, but an exponential may be infinite there
#pragma unroll 1
          for (int c = 0; c < n_last; c += 16) {
            uint32_t sv[16], dv[16], pk[8];
            tmem_ld16(tS + c, sv);
            tmem_ld16(tdP + c, dv);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float p0 = mufu_exp2(fmaf(__uint_as_float(sv[2 * i]), p.scale_log2, nlse));
              const float p1 = mufu_exp2(fmaf(__uint_as_float(sv[2 * i + 1]), p.scale_log2, nlse));
              float d0 = p0 * (__uint_as_float(dv[2 * i]) + ndelta);
              float d1 = p1 * (__uint_as_float(dv[2 * i + 1]) + ndelta);
              if (c + 2 * i >= rem) d0 = 0.f;
              if (c + 2 * i + 1 >= rem) d1 = 0.f;
              pk[i] = pack_bf16x2(d0, d1);
            }
            tmem_st8(tS + (c >> 1), pk);
          }
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&next_full[wg]);
        if (pending) {
          pending = false;
          if (!epilogue(it - 1)) { ok = false; break; }
        }
      }
      if (!ok) break;
      if (pending && !epilogue(it - 1)) { ok = false; break; }
      j -= nkv;                        // the stream of tiles runs on into the next item
    }
    if (ok) epilogue(n_items - 1);
    if (R::STAGED) out.drain();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

template <int DCH>
__global__ void __launch_bounds__(128 + 128 * BwdRing<DCH>::NWG, 1)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
                    const __grid_constant__ CUtensorMap tm_dk, const __grid_constant__ CUtensorMap tm_dv,
                    const AttnBwdParams p, const int n_items_total) {
  using R = BwdRing<DCH>;
  constexpr int HD = 64 * DCH;
  constexpr int KB = DCH * 16384;  // K tile, V tile (128 rows)
  constexpr int QB = DCH * 8192;   // Q tile, dO tile (64 rows)
  constexpr int NWG = R::NWG, NST = R::NST, NB = R::NB;
  static_assert(NWG * 128 + 2 * HD <= 512, "TMEM columns");
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sKV = smem;                   // [NB] items: K | V
  uint8_t* sQD = sKV + NB * R::ITEM_BYTES;                          // [NST] Q | dO
  uint8_t* sOut = sQD + NST * R::STAGE;                             // [NWG]
  float* s_stat = reinterpret_cast<float*>(sOut + NWG * R::OUT_BYTES);   // [NST] lse [64] | delta [64]
  uint64_t* bars = reinterpret_cast<uint64_t*>(s_stat + R::STAT);
  uint64_t* kv_full = bars;              // [NB <= 2]
  uint64_t* kv_empty = bars + 2;         // [NB]
  uint64_t* first_full = bars + 4;       // [NWG <= 3] Q, dO and their row statistics for the first tile of each chain
  uint64_t* next_full = bars + 7;        // [NWG] P and dS of the chain's tile are in TMEM, its next tile has landed
  uint64_t* qd_empty = bars + 10;        // [NST <= 6]
  uint64_t* sp_full = bars + 16;         // [NWG]
  uint64_t* acc_full = bars + 19;
  uint64_t* acc_empty = bars + 20;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 21);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int N = p.N;
  const int nfull = N / BT, rem = N - nfull * BT;
  const int nq = nfull + (rem ? 1 : 0);
  const int n_last = rem ? ((rem + 15) & ~15) : BT;
  const int row_tiles = (N + TILE - 1) / TILE;
  const int n_ctas = static_cast<int>(gridDim.x);
  const int n_items = (n_items_total - static_cast<int>(blockIdx.x) + n_ctas - 1) / n_ctas;

  if (threadIdx.x == 0) {
    int ab = (p.status && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
    if ((smem_u32(smem) & 1023u) != 0) { ab = 1; if (p.status) atomicCAS(p.status, 0, ERR_BOUNDS); }
    *s_abort = ab;
  }
  __syncthreads();
  if (*s_abort) return;
  if (threadIdx.x == 0) {
    prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v); prefetch_tmap(&tm_do);
    for (int i = 0; i < NB; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < NST; ++i) mbar_init(&qd_empty[i], 1);
    // a tile's arrivals: the TMA loads and 32 lanes of row statistics (plus, from the second round on, four math warps)
    for (int i = 0; i < NWG; ++i) {
      mbar_init(&first_full[i], 1 + 32);
      mbar_init(&next_full[i], 4 + 1 + 32);
      mbar_init(&sp_full[i], 1);
    }
    mbar_init(acc_full, 1); mbar_init(acc_empty, 4 * NWG);
    fence_barrier_init();
  }
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tdK = tmem_base + NWG * 128, tdV = tdK + HD;     // chain w: S^T at w * 128, dP^T at w * 128 + 64

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one_sync()) {
      auto load_item = [&](int it) -> bool {
        const int b = it % NB;
        if (!mbar_wait(&kv_empty[b], ((it / NB) & 1) ^ 1, p.status, ERR_TIMEOUT_ATTN)) return false;
        const BwdItem w = bwd_item(it, row_tiles, p.H);
        mbar_expect_tx(&kv_full[b], R::ITEM_BYTES);
        uint8_t* d = sKV + b * R::ITEM_BYTES;
#pragma unroll
        for (int c = 0; c < DCH; ++c) {
          tma_load_4d(d + c * 16384, &tm_k, &kv_full[b], c * 64, w.head, w.tile * TILE, w.win);
          tma_load_4d(d + KB + c * 16384, &tm_v, &kv_full[b], c * 64, w.head, w.tile * TILE, w.win);
        }
        return true;
      };
      bool ok = load_item(0);
      int st = 0, t = 0;
      uint32_t ph = 1;
      // where an item's own operands are requested: with two buffers those of the next item early in this one, with one
      // buffer those of this item behind its first tiles (they have to wait for the last scores of the item before)
      const int j_item = min(NB == 2 ? 2 : NWG - 1, nq - 1);
      for (int it = 0; it < n_items && ok; ++it) {
        const BwdItem w = bwd_item(it, row_tiles, p.H);
        for (int j = 0; j < nq; ++j, ++t) {
          if (!mbar_wait(&qd_empty[st], ph, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
          uint64_t* bar = t < NWG ? &first_full[t] : &next_full[t % NWG];
          uint8_t* d = sQD + st * R::STAGE;
          mbar_expect_tx(bar, R::STAGE);
#pragma unroll
          for (int c = 0; c < DCH; ++c) {
            tma_load_4d(d + c * 8192, &tm_q, bar, c * 64, w.head, j * BT, w.win);
            tma_load_4d(d + QB + c * 8192, &tm_do, bar, c * 64, w.head, j * BT, w.win);
          }
          if (++st == NST) { st = 0; ph ^= 1; }
          if (j == j_item) {
            if (NB == 2 && it + 1 < n_items && !load_item(it + 1)) { ok = false; break; }
            if (NB == 1 && it > 0 && !load_item(it)) { ok = false; break; }
          }
        }
      }
      // the last tile of each chain has no successor: its round completes without loads
      for (int e = t + NWG; t < e && ok; ++t) {
        if (!mbar_wait(&qd_empty[st], ph, p.status, ERR_TIMEOUT_ATTN)) break;
        if (t >= NWG) mbar_arrive(&next_full[t % NWG]);
        if (++st == NST) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (elect_one_sync()) {
      const uint32_t aI = smem_u32(sKV), aS = smem_u32(sQD);
      const int total = n_items * nq;
      TileIter s;                       // next tile whose scores are issued
      int s_w = 0, s_st = 0;
      // S^T = K Q_j^T and dP^T = V dO_j^T of tile s
      auto issue_sp = [&]() -> bool {
        const int b = s.it % NB;
        if (s.j == 0) {
          if (!mbar_wait(&kv_full[b], (s.it / NB) & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
          tc_fence_after();
        }
        const bool last = s.j == nq - 1;
        const uint32_t idesc = make_idesc_bf16(TILE, last ? n_last : BT, 0, 0);
        const uint32_t tS = tmem_base + s_w * 128;
        const uint64_t d0 = make_smem_desc(aI + b * R::ITEM_BYTES, 0, 1024), d1 = d0 + KB / 16;
        const uint64_t d2 = make_smem_desc(aS + s_st * R::STAGE, 0, 1024), d3 = d2 + QB / 16;
#pragma unroll
        for (int kk = 0; kk < 4 * DCH; ++kk)
          umma_ss(tS, d0 + ((kk >> 2) * 16384 + (kk & 3) * 32) / 16, d2 + ((kk >> 2) * 8192 + (kk & 3) * 32) / 16, idesc,
                  kk > 0);
#pragma unroll
        for (int kk = 0; kk < 4 * DCH; ++kk)
          umma_ss(tS + 64, d1 + ((kk >> 2) * 16384 + (kk & 3) * 32) / 16, d3 + ((kk >> 2) * 8192 + (kk & 3) * 32) / 16,
                  idesc, kk > 0);
        tc_commit(&sp_full[s_w]);
        if (last) tc_commit(&kv_empty[b]);
        if (++s_w == NWG) s_w = 0;
        if (++s_st == NST) s_st = 0;
        s.next(nq);
        return true;
      };
      bool ok = true;
      for (int i = 0; i < NWG && i < total && ok; ++i) {
        ok = mbar_wait(&first_full[i], 0, p.status, ERR_TIMEOUT_ATTN);
        tc_fence_after();
        if (ok) ok = issue_sp();
      }
      int w = 0, st = 0;
      uint32_t ph = 0;
      TileIter a;
      constexpr uint32_t idesc_acc = make_idesc_bf16(TILE, HD, 0, 1);
      while (ok && a.g < total) {
        if (!mbar_wait(&next_full[w], ph, p.status, ERR_TIMEOUT_ATTN)) break;
        if (a.j == 0 && a.it > 0 && !mbar_wait(acc_empty, (a.it - 1) & 1, p.status, ERR_TIMEOUT_ATTN)) break;
        tc_fence_after();
        const bool last = a.j == nq - 1;
        const uint32_t acc0 = a.j > 0 ? 1u : 0u;
        const uint32_t tA = tmem_base + w * 128;
        // dV += P^T dO_j, dK += dS^T Q_j : A from TMEM (16 q columns = 8 words per K step), B MN-major (d contiguous)
        const uint64_t dq = make_smem_desc(aS + st * R::STAGE, 8192, 1024), dg = dq + QB / 16;
        if (!last || rem == 0) {
#pragma unroll
          for (int kk = 0; kk < BT / 16; ++kk) umma_ts(tdV, tA + kk * 8, dg + kk * 128, idesc_acc, kk ? 1u : acc0);
#pragma unroll
          for (int kk = 0; kk < BT / 16; ++kk) umma_ts(tdK, tA + 64 + kk * 8, dq + kk * 128, idesc_acc, kk ? 1u : acc0);
        } else {
          for (int kk = 0; kk < n_last / 16; ++kk) umma_ts(tdV, tA + kk * 8, dg + kk * 128, idesc_acc, kk ? 1u : acc0);
          for (int kk = 0; kk < n_last / 16; ++kk) umma_ts(tdK, tA + 64 + kk * 8, dq + kk * 128, idesc_acc, kk ? 1u : acc0);
        }
        tc_commit(&qd_empty[st]);
        if (last) tc_commit(acc_full);
        // the tensor core executes in issue order: these scores overwrite the A operand above only after it was read
        if (s.g < total && !issue_sp()) break;
        if (++w == NWG) { w = 0; ph ^= 1; }
        if (++st == NST) st = 0;
        a.next(nq);
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------ lse and delta of the rows of every streamed tile
    // (asynchronous 4-byte copies: a window's first row need not be 16-byte aligned; rows past its end become zeros)
    int st = 0, t = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (int it = 0; it < n_items && ok; ++it) {
      const BwdItem w = bwd_item(it, row_tiles, p.H);
      const size_t sbase = (static_cast<size_t>(w.win) * p.H + w.head) * N;
      for (int j = 0; j < nq; ++j, ++t) {
        if (!mbar_wait(&qd_empty[st], ph, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
        float* d = s_stat + st * 2 * BT + lane;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int r = j * BT + u * 32 + lane;
          const uint32_t bytes = (r < N) ? 4u : 0u;
          const size_t src = sbase + (r < N ? r : 0);
          cp_async4(d + u * 32, p.lse + src, bytes);
          cp_async4(d + BT + u * 32, p.delta + src, bytes);
        }
        cp_async_arrive(t < NWG ? &first_full[t] : &next_full[t % NWG]);
        if (++st == NST) { st = 0; ph ^= 1; }
      }
    }
    for (int e = t + NWG; t < e && ok; ++t) {
      if (!mbar_wait(&qd_empty[st], ph, p.status, ERR_TIMEOUT_ATTN)) break;
      if (t >= NWG) mbar_arrive(&next_full[t % NWG]);
      if (++st == NST) { st = 0; ph ^= 1; }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp >= 4) {
    // ------------------------------------------------------------ math: one thread = one K/V row, every NWG-th tile
    const int wg = (warp >> 2) - 1, q = warp & 3;
    const int row = q * 32 + lane;  // kv row within the tile
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t tS = tmem_base + lane_addr + wg * 128, tdP = tS + 64;
    const uint64_t nsl = f2_pack(-p.scale_log2, -p.scale_log2);
    const float sc = p.scale;
    uint32_t ph = 0;
    int j = wg, g = wg;
    bool ok = true;
    // Columns past the window's end have zero Q and dO rows and zero statistics (P = 1, dS = 0): they add nothing. Rows
    // past its end may hold anything: they are not stored.
    auto pair = [&](uint32_t s0, uint32_t s1, uint32_t d0, uint32_t d1, uint64_t l, uint64_t de, uint32_t& pp,
                    uint32_t& dd) {
      float t0, t1;
      f2_unpack(f2_fma(f2_pack(__uint_as_float(s0), __uint_as_float(s1)), nsl, l), t0, t1);     // -(log2 P)
      const uint64_t pr = f2_pack(mufu_exp2(-t0), mufu_exp2(-t1));
      pp = f2_to_bf16x2(pr);
      dd = f2_to_bf16x2(f2_mul(pr, f2_sub(f2_pack(__uint_as_float(d0), __uint_as_float(d1)), de)));
    };
    BwdOut out{sOut + wg * R::OUT_BYTES + q * 4096, lane, q * 32};
    // see attn_bwd_dq_kernel: the epilogue of an item runs after this warpgroup's first tile of the next
    auto epilogue = [&](int it) -> bool {
      if (!mbar_wait(acc_full, it & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
      tc_fence_after();
      const BwdItem w = bwd_item(it, row_tiles, p.H);
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty);
      };
      if (R::STAGED && p.push_n_local == 0) {
        int mine = 0;                   // this warpgroup's groups of 32 columns of dK and dV
        for (int c = wg * 32; c < 2 * HD; c += 32 * NWG) mine += (c < HD ? c : c - HD) < p.d;
        if (mine == 0) release();
        for (int c = wg * 32; c < 2 * HD; c += 32 * NWG) {
          const int col = c < HD ? c : c - HD;          // column inside the head
          if (col < p.d)
            out.put(tdK + lane_addr + c, c < HD ? sc : 1.f, c < HD ? &tm_dk : &tm_dv, col, w.head, w.tile * TILE, w.win, N,
                    [&] { if (--mine == 0) release(); });
        }
        return true;
      }
      const int grow = w.tile * TILE + row;
      const bool row_ok = grow < N;
      __nv_bfloat16* dk = bwd_dst(p, w.win, row_ok ? grow : 0, w.head, 1, p.k_col0);
      __nv_bfloat16* dv = bwd_dst(p, w.win, row_ok ? grow : 0, w.head, 2, p.v_col0);
#pragma unroll
      for (int c = 0; c < 2 * HD; c += 32) {
        const int col = c < HD ? c : c - HD;            // column inside the head
        if ((c / 32) % NWG != wg || col >= p.d) continue;
        uint32_t v[32];
        tmem_ld32(tdK + lane_addr + c, v);
        tmem_wait_ld();
        __nv_bfloat16* dst = ((c < HD) ? dk : dv) + col;
        const float f = (c < HD) ? sc : 1.f;
        if (row_ok) {
#pragma unroll
          for (int gq = 0; gq < 4; ++gq) {
            uint32_t o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              o[i] = pack_bf16x2(__uint_as_float(v[8 * gq + 2 * i]) * f, __uint_as_float(v[8 * gq + 2 * i + 1]) * f);
            if (col + gq * 8 < p.d) *reinterpret_cast<uint4*>(dst + gq * 8) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(acc_empty);
      return true;
    };
    for (int it = 0; it < n_items && ok; ++it) {
      bool pending = it > 0;
      for (; j < nq; j += NWG, g += NWG, ph ^= 1) {
        const int st = g % NST;
        if (!mbar_wait(&sp_full[wg], ph, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
        tc_fence_after();
        const ulonglong2* ls = reinterpret_cast<const ulonglong2*>(s_stat + st * 2 * BT);
        const ulonglong2* ds = ls + BT / 4;
        if (j < nfull) {
#pragma unroll
          for (int c = 0; c < 64; c += 32) {
            uint32_t sv[32], dv[32], pp[16], dd[16];
            tmem_ld32(tS + c, sv);
            tmem_ld32(tdP + c, dv);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const ulonglong2 l = ls[c / 4 + i], de = ds[c / 4 + i];
              pair(sv[4 * i], sv[4 * i + 1], dv[4 * i], dv[4 * i + 1], l.x, de.x, pp[2 * i], dd[2 * i]);
              pair(sv[4 * i + 2], sv[4 * i + 3], dv[4 * i + 2], dv[4 * i + 3], l.y, de.y, pp[2 * i + 1], dd[2 * i + 1]);
            }
            tmem_st16(tS + (c >> 1), pp);
            tmem_st16(tdP + (c >> 1), dd);
          }
        } else {
#pragma unroll 1
          for (int c = 0; c < n_last; c += 16) {
            uint32_t sv[16], dv[16], pp[8], dd[8];
            tmem_ld16(tS + c, sv);
            tmem_ld16(tdP + c, dv);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const ulonglong2 l = ls[c / 4 + i], de = ds[c / 4 + i];
              pair(sv[4 * i], sv[4 * i + 1], dv[4 * i], dv[4 * i + 1], l.x, de.x, pp[2 * i], dd[2 * i]);
              pair(sv[4 * i + 2], sv[4 * i + 3], dv[4 * i + 2], dv[4 * i + 3], l.y, de.y, pp[2 * i + 1], dd[2 * i + 1]);
            }
            tmem_st8(tS + (c >> 1), pp);
            tmem_st8(tdP + (c >> 1), dd);
          }
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&next_full[wg]);
        if (pending) {
          pending = false;
          if (!epilogue(it - 1)) { ok = false; break; }
        }
      }
      if (!ok) break;
      if (pending && !epilogue(it - 1)) { ok = false; break; }
      j -= nq;                        // the stream of tiles runs on into the next item
    }
    if (ok) epilogue(n_items - 1);
    if (R::STAGED) out.drain();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, 512);
}

template <int DCH>
static int launch_attn_bwd(const CUtensorMap& tq128, const CUtensorMap& tk64, const CUtensorMap& tv64,
                           const CUtensorMap& tdo128, const CUtensorMap& tq64, const CUtensorMap& tk128,
                           const CUtensorMap& tv128, const CUtensorMap& tdo64, const CUtensorMap (&out)[3],
                           const AttnBwdParams& p, cudaStream_t stream) {
  using R = BwdRing<DCH>;
  auto k1 = attn_bwd_dq_kernel<DCH>;
  auto k2 = attn_bwd_dkv_kernel<DCH>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, R::SMEM) != cudaSuccess) return -20;
    if (cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, R::SMEM) != cudaSuccess) return -20;
    configured = true;
  }
  const long long items = static_cast<long long>((p.N + TILE - 1) / TILE) * p.H * p.n_win;
  if (items > 0x3fffffff) return -23;
  const int n = static_cast<int>(items), grid = n < num_sms() ? n : num_sms();
  k1<<<grid, R::THREADS, R::SMEM, stream>>>(tq128, tk64, tv64, tdo128, out[0], p, n);
  if (cudaGetLastError() != cudaSuccess) return -21;
  k2<<<grid, R::THREADS, R::SMEM, stream>>>(tq64, tk128, tv128, tdo64, out[1], out[2], p, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -22;
}

}  // namespace aeris

using namespace aeris;

// Variant of the forward kernel. poly (head_dim 64 only): -1 = scalar softmax arithmetic, exp unit only; 0 = two-wide
// fp32 arithmetic; 2 = two-wide with two of every eight score pairs on the polynomial exp2. mode: see AttnFwdRing
// (0 probabilities through shared memory; 1 in tensor memory; 2 in tensor memory, four CTAs per SM).
static int g_fwd_poly = -1;
static int g_fwd_mode = 0;
extern "C" int aeris_attn_set_fwd_variant(int poly, int mode) {
  if ((poly != -1 && poly != 0 && poly != 2) || mode < 0 || mode > 2) return -1;
  g_fwd_poly = poly;
  g_fwd_mode = mode;
  return 0;
}
#ifdef AERIS_ATTN_TRACE
extern "C" int aeris_attn_set_trace(long long* buf) {
  return cudaMemcpyToSymbol(aeris::g_attn_trace, &buf, sizeof(buf)) == cudaSuccess ? 0 : -1;
}
#endif
extern "C" int aeris_attn_set_fwd_smem_pad(int bytes) {
  if (bytes < 0 || bytes > 160 * 1024) return -1;
  g_fwd_smem_pad = bytes;
  return 0;
}

// The kernels read and write o, d_o and dqkv in 16-byte vectors: bases on 16-byte boundaries, pitches and column offsets
// (`elems`: their bitwise or) in whole vectors of eight elements. q, k and v are checked where their tensor maps are made.
static bool whole_vectors(const void* base, int elems) {
  return (reinterpret_cast<uintptr_t>(base) & 15) == 0 && (elems & 7) == 0;
}

// q, k, v: base pointers of row-major [n_win * N, ld*] bf16 tensors; *_col0 = column of head 0.
static int attn_fwd_impl(const void* q, int ldq, int q_col0, const void* k, int ldk, int k_col0, const void* v,
                         int ldv, int v_col0, void* o, int ldo, float* lse, int n_win, int N, int H, int head_dim,
                         float scale, int* status, void* stream_, const void* const* o_peers, int sp,
                         int push_n_local, int push_ld, int push_col0);

extern "C" int aeris_attn_fwd(const void* q, int ldq, int q_col0, const void* k, int ldk, int k_col0, const void* v,
                              int ldv, int v_col0, void* o, int ldo, float* lse, int n_win, int N, int H,
                              int head_dim, float scale, int* status, void* stream_) {
  return attn_fwd_impl(q, ldq, q_col0, k, ldk, k_col0, v, ldv, v_col0, o, ldo, lse, n_win, N, H, head_dim, scale, status,
                       stream_, nullptr, 0, 0, 0, 0);
}

// Forward whose output rows are (also) pushed to the ranks that own the tokens (Ulysses return exchange fused into the
// attention epilogue). `o` may be null when only the pushed copy is wanted. head_dim 64 or 128.
extern "C" int aeris_attn_fwd_push(const void* qkv, int ld, int H_local, void* o, int ldo, float* lse, int n_win, int N,
                                   int head_dim, float scale, const void* const* o_peers, int sp, int n_local,
                                   int push_ld, int push_col0, int* status, void* stream_) {
  if (head_dim != 64 && head_dim != 128) return -1;
  const int hd = H_local * head_dim;
  return attn_fwd_impl(qkv, ld, 0, qkv, ld, hd, qkv, ld, 2 * hd, o, ldo, lse, n_win, N, H_local, head_dim, scale,
                       status, stream_, o_peers, sp, n_local, push_ld, push_col0);
}

static int attn_fwd_impl(const void* q, int ldq, int q_col0, const void* k, int ldk, int k_col0, const void* v,
                         int ldv, int v_col0, void* o, int ldo, float* lse, int n_win, int N, int H, int head_dim,
                         float scale, int* status, void* stream_, const void* const* o_peers, int sp,
                         int push_n_local, int push_ld, int push_col0) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (head_dim <= 0 || head_dim > 128 || head_dim % 8) return -1;
  if (n_win <= 0 || N <= 0 || H <= 0 || n_win > 65535 || H > 65535) return -2;
  if (sp < 0 || sp > 8 || (!o && !o_peers)) return -3;
  if (!whole_vectors(o, ldo)) return -4;
  for (int i = 0; i < sp; ++i)
    if (!whole_vectors(o_peers[i], push_ld | push_col0)) return -4;
  AttnFwdParams p{};
  for (int i = 0; i < sp; ++i) p.o_peers[i] = const_cast<void*>(o_peers[i]);
  p.push_n_local = o_peers ? push_n_local : 0; p.push_ld = push_ld; p.push_col0 = push_col0;
  p.O = reinterpret_cast<__nv_bfloat16*>(o); p.ldo = ldo; p.lse = lse; p.N = N; p.H = H; p.n_win = n_win;
  p.d = head_dim;
  p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
  CUtensorMap tq, tk, tv;
  int r;
  auto at = [](const void* base, int col) -> const void* { return reinterpret_cast<const __nv_bfloat16*>(base) + col; };
  if ((r = make_tmap_heads_bf16(&tq, at(q, q_col0), head_dim, H, N, n_win, ldq, TILE))) return r;
  // Two query tiles at a time where there are two; its masked columns need a positive scale. ms, windows x tokens, one tile
  // at a time / two in turn, 24 heads x 64 and 12 x 128:
  // - Three or five tiles of which the last is not full leave the second chain idle for a third or a fifth of the time.
  //   64-wide heads are faster without then (249 x 260 tokens 0.387 / 0.416, 202 x 320 0.348 / 0.352, 221 x 513 0.857 /
  //   0.925, 175 x 576 0.732 / 0.772; full ones 168 x 384 0.363 / 0.337, 142 x 640 0.689 / 0.664; seven tiles 84 x 832 0.692
  //   / 0.667, 97 x 772 0.758 / 0.754), 128-wide ones are not (249 x 260 0.325 / 0.295, 175 x 576 0.621 / 0.550).
  // - A last half tile that is cut off (CUT) costs every tile: short windows only. 64: 240 tokens 0.295 / 0.243, 500 0.458 /
  //   0.393, 740 0.726 / 0.689, 970 0.661 / 0.680, 1250 0.635 / 0.624, 1500 0.588 / 0.605, 3600 0.498 / 0.538. 128: 740
  //   0.577 / 0.458, 1250 0.481 / 0.423, 1500 0.441 / 0.421, 2000 0.417 / 0.423, 3600 0.360 / 0.372.
  const int q_tiles = (N + TILE - 1) / TILE;
  const bool idle_chain = head_dim <= 64 && (q_tiles == 3 || q_tiles == 5) && N % TILE != 0;
  const bool cut = N % KVT > 4, long_cut = cut && q_tiles > (head_dim > 64 ? 12 : 6);
  if (q_tiles > 1 && !idle_chain && !long_cut && scale > 0.f && g_fwd_mode == 0 && g_fwd_poly == -1) {
    if ((r = make_tmap_heads_bf16(&tk, at(k, k_col0), head_dim, H, N, n_win, ldk, KVP))) return r;
    if ((r = make_tmap_heads_bf16(&tv, at(v, v_col0), head_dim, H, N, n_win, ldv, KVP))) return r;
    CUtensorMap to = tq;      // without a local output nothing is stored through it
    if (o && (r = make_tmap_heads_bf16(&to, o, head_dim, H, N, n_win, ldo, 32))) return r;
    if (cut)
      return head_dim > 64 ? launch_attn_fwd_pair<2, true>(tq, tk, tv, to, p, stream)
                           : launch_attn_fwd_pair<1, true>(tq, tk, tv, to, p, stream);
    return head_dim > 64 ? launch_attn_fwd_pair<2, false>(tq, tk, tv, to, p, stream)
                         : launch_attn_fwd_pair<1, false>(tq, tk, tv, to, p, stream);
  }
  if ((r = make_tmap_heads_bf16(&tk, at(k, k_col0), head_dim, H, N, n_win, ldk, KVT))) return r;
  if ((r = make_tmap_heads_bf16(&tv, at(v, v_col0), head_dim, H, N, n_win, ldv, KVT))) return r;
  if (head_dim > 64) {
    switch (g_fwd_mode) {
      case 1: return launch_attn_fwd<2, -1, 1>(tq, tk, tv, p, stream);
      default: return launch_attn_fwd<2, -1, 0>(tq, tk, tv, p, stream);
    }
  }
  const bool poly = g_fwd_poly == 2;
  switch (g_fwd_mode) {
    case 1: return poly ? launch_attn_fwd<1, 2, 1>(tq, tk, tv, p, stream) : launch_attn_fwd<1, -1, 1>(tq, tk, tv, p, stream);
    case 2: return launch_attn_fwd<1, -1, 2>(tq, tk, tv, p, stream);
    default: break;
  }
  if (g_fwd_poly == 0) return launch_attn_fwd<1, 0, 0>(tq, tk, tv, p, stream);
  return poly ? launch_attn_fwd<1, 2, 0>(tq, tk, tv, p, stream) : launch_attn_fwd<1, -1, 0>(tq, tk, tv, p, stream);
}

// Backward. qkv: fused [T, ldq] tensor (q/k/v column blocks at *_col0); o, d_o: [T, ldo]; dqkv: [T, ldg] (same
// column layout as qkv); lse from the forward; delta: scratch [n_win*H*N] fp32 written by the first kernel.
static int attn_bwd_impl(const void* qkv, int ldq, int q_col0, int k_col0, int v_col0, const void* o, const void* d_o,
                         int ldo, const float* lse, float* delta, void* dqkv, int ldg, int n_win, int N, int H,
                         int head_dim, float scale, int* status, void* stream_, const void* const* dq_peers, int sp,
                         int push_n_local, int push_ld, int push_sec_w, int push_col0);

extern "C" int aeris_attn_bwd(const void* qkv, int ldq, int q_col0, int k_col0, int v_col0, const void* o,
                              const void* d_o, int ldo, const float* lse, float* delta, void* dqkv, int ldg,
                              int n_win, int N, int H, int head_dim, float scale, int* status, void* stream_) {
  return attn_bwd_impl(qkv, ldq, q_col0, k_col0, v_col0, o, d_o, ldo, lse, delta, dqkv, ldg, n_win, N, H, head_dim,
                       scale, status, stream_, nullptr, 0, 0, 0, 0, 0);
}

// Backward whose dQ / dK / dV rows are pushed to the ranks that own the tokens (layout [tokens_local, 3 * heads * d]).
// head_dim 64 or 128.
extern "C" int aeris_attn_bwd_push(const void* qkv, int ld, int H_local, const void* o, const void* d_o, int ldo,
                                   const float* lse, float* delta, int n_win, int N, int head_dim, float scale,
                                   const void* const* dq_peers, int sp, int n_local, int push_ld, int push_sec_w,
                                   int push_col0, int* status, void* stream_) {
  if (head_dim != 64 && head_dim != 128) return -1;
  const int hd = H_local * head_dim;
  return attn_bwd_impl(qkv, ld, 0, hd, 2 * hd, o, d_o, ldo, lse, delta, nullptr, 0, n_win, N, H_local, head_dim, scale,
                       status, stream_, dq_peers, sp, n_local, push_ld, push_sec_w, push_col0);
}

static int attn_bwd_impl(const void* qkv, int ldq, int q_col0, int k_col0, int v_col0, const void* o, const void* d_o,
                         int ldo, const float* lse, float* delta, void* dqkv, int ldg, int n_win, int N, int H,
                         int head_dim, float scale, int* status, void* stream_, const void* const* dq_peers, int sp,
                         int push_n_local, int push_ld, int push_sec_w, int push_col0) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (head_dim <= 0 || head_dim > 128 || head_dim % 8) return -1;
  if (n_win <= 0 || N <= 0 || H <= 0 || n_win > 65535 || H > 65535) return -2;
  if (sp < 0 || sp > 8 || (!dqkv && !dq_peers)) return -3;
  if (!whole_vectors(o, ldo) || !whole_vectors(d_o, ldo) || !whole_vectors(dqkv, ldg | q_col0 | k_col0 | v_col0)) return -4;
  for (int i = 0; i < sp; ++i)
    if (!whole_vectors(dq_peers[i], push_ld | push_sec_w | push_col0)) return -4;
  AttnBwdParams p{};
  for (int i = 0; i < sp; ++i) p.dq_peers[i] = const_cast<void*>(dq_peers[i]);
  p.push_n_local = dq_peers ? push_n_local : 0; p.push_ld = push_ld; p.push_sec_w = push_sec_w; p.push_col0 = push_col0;
  p.O = reinterpret_cast<const __nv_bfloat16*>(o); p.dO = reinterpret_cast<const __nv_bfloat16*>(d_o); p.ldo = ldo;
  p.lse = lse; p.delta = delta; p.dQKV = reinterpret_cast<__nv_bfloat16*>(dqkv); p.ldg = ldg;
  p.N = N; p.H = H; p.n_win = n_win; p.d = head_dim; p.q_col0 = q_col0; p.k_col0 = k_col0; p.v_col0 = v_col0;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.status = status;
  CUtensorMap q128, q64, k128, k64, v128, v64, d128, d64;
  int r;
  const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(qkv);
  const struct { CUtensorMap* m; const void* base; int ld; uint32_t rows; } maps[] = {
      {&q128, b + q_col0, ldq, TILE}, {&q64, b + q_col0, ldq, BT},
      {&k128, b + k_col0, ldq, TILE}, {&k64, b + k_col0, ldq, BT},
      {&v128, b + v_col0, ldq, TILE}, {&v64, b + v_col0, ldq, BT},
      {&d128, d_o, ldo, TILE},        {&d64, d_o, ldo, BT}};
  for (const auto& m : maps)
    if ((r = make_tmap_heads_bf16(m.m, m.base, head_dim, H, N, n_win, m.ld, m.rows))) return r;
  CUtensorMap out[3] = {q128, q128, q128};      // pushed gradients and those of narrow heads do not leave through them
  if (head_dim > 64 && !dq_peers) {
    const __nv_bfloat16* g = p.dQKV;
    const int cols[3] = {q_col0, k_col0, v_col0};
    for (int i = 0; i < 3; ++i)
      if ((r = make_tmap_heads32_bf16(&out[i], g + cols[i], head_dim, H, N, n_win, ldg, 32))) return r;
  }
  return head_dim <= 64 ? launch_attn_bwd<1>(q128, k64, v64, d128, q64, k128, v128, d64, out, p, stream)
                        : launch_attn_bwd<2>(q128, k64, v64, d128, q64, k128, v128, d64, out, p, stream);
}

// ------------------------------------------------------------------------------------------ allocation-free variant
// Same computation as aeris_attn_bwd, for hosts that must not allocate device memory at call time (declared and
// described in noalloc.h). The `delta` scratch (one float per (window, head, token)) lives in this file-scope device
// array instead of a caller-provided buffer. The array name is only a host-side handle: its device address is
// looked up once per device with cudaGetSymbolAddress and that address is what the kernels receive.
#include "noalloc.h"

static __device__ __align__(256) float g_attn_delta_scratch[AERIS_NOALLOC_MAX_SCRATCH_FLOATS];
static float* g_attn_delta_ptr[AERIS_NOALLOC_MAX_DEVICES] = {};

extern "C" int aeris_attn_bwd_noalloc(const void* qkv, int ldq, int q_col0, int k_col0, int v_col0, const void* o,
                                      const void* d_o, int ldo, const float* lse, void* dqkv, int ldg, int n_win,
                                      int N, int H, int head_dim, float scale, int* status, void* stream_) {
  if (n_win <= 0 || N <= 0 || H <= 0) return AERIS_NOALLOC_ERR_BAD_SHAPE;
  const long long need = static_cast<long long>(n_win) * H * N;
  if (need > AERIS_NOALLOC_MAX_SCRATCH_FLOATS) return AERIS_NOALLOC_ERR_TOO_LARGE;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= AERIS_NOALLOC_MAX_DEVICES)
    return AERIS_NOALLOC_ERR_DEVICE;
  if (g_attn_delta_ptr[dev] == nullptr) {
    // one-time set-up for this device (which is current): resolve the device address of the scratch array
    float* ptr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_attn_delta_scratch);
    if (e != cudaSuccess || ptr == nullptr) return AERIS_NOALLOC_ERR_SYMBOL;
    g_attn_delta_ptr[dev] = ptr;
  }
  return aeris_attn_bwd(qkv, ldq, q_col0, k_col0, v_col0, o, d_o, ldo, lse, g_attn_delta_ptr[dev], dqkv, ldg, n_win,
                        N, H, head_dim, scale, status, stream_);
}
