// Attention backward. Included by attention.cu. Two kernels, neither needs atomics; in both an item is a 128-row tile of one
// (window, head) with two operands I0, I1 of its own, and two operands R0, R1 are streamed past it in tiles of BT rows:
//   dQ    (DKV = false): I0 = Q, I1 = dO, R0 = K, R1 = V. S = Q K^T, dP = dO V^T, dS = P * (dP - delta),
//                        dQ = scale * sum dS K. Also writes delta = rowsum(dO * O).
//   dK/dV (DKV = true) : I0 = K, I1 = V, R0 = Q, R1 = dO. S^T = K Q^T, dP^T = V dO^T, dV = sum P^T dO,
//                        dK = scale * sum dS^T Q.
//
// One persistent CTA per SM. Two chains take the streamed tiles in turn, each with TMEM columns of its own for S and dP; P
// and dS go back into the columns they came from and are the A operand of the accumulating products from there. A chain's
// next scores are issued as soon as its last ones have been read (dQ) or turned into P (dK/dV), its next dP behind the
// product that takes dS, so that both are computed under arithmetic. Two warps issue products, each in its own order: A the
// scores and dV, B dP and dQ or dK. Two warpgroups share a chain's tile, half of the columns each, because what bounds the
// math warps is the latency of their own steps, not a unit; another warpgroup takes the gradients to memory, so that no
// math warp waits for an item's last products. A chain's round of 2,300 cycles at head_dim 64 (96 columns) is 1,070 of
// exponentials (768 by themselves), 440 of dS and 500-800 of waits; ncu, 36 windows of 900 tokens, dQ and dK/dV: tensor core
// at 48 and 56 %, exponential unit at 65 and 56.
// At 128 the products bound it: 64-column tiles (a wider one has no room in shared memory) take 48 cycles per step of 16
// where 32 would be the rate, because both operands come from shared memory.
//
// Both kernels, ms, one call, bursts of 6 ms, with one issuer and 64 columns per chain and warpgroup / now: 72 windows x 900
// tokens, 24 heads x 64 1.73 / 1.41; 12 x 128 1.42 / 1.24; 16 x 3600, 12 x 128 3.80 / 3.40; 200 x 225, 24 x 64
// 0.645 / 0.488, 12 x 128 0.534 / 0.465; 400 x 64, 24 x 64 0.436 / 0.349; 8 x 900, 4 x 64 0.0522 / 0.0457.
// On the way: three chains of 64 columns and one warpgroup each 1.57, with 32-column halves in a rolled loop 1.62; the
// issuers' loops unrolled over the ring 2.45 (instruction cache); single threads as issuers 1.446 for 1.432 (128: 1.333
// for 1.260); waits with a call behind the first try 1.65; turns at the exponentials 1.83 for 1.57.
#pragma once
#include <stddef.h>

namespace aeris {

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

// Shared memory (227 KB) and the 512 TMEM columns set the numbers: the chains' S and dP + the accumulators (HD columns for
// dQ, twice while there is room; HD each for dK and dV).
template <int DCH, bool DKV> struct BwdCfg {
  static constexpr int HD = 64 * DCH;
  static constexpr int BT = (DCH == 1) ? 96 : 64;         // rows of a streamed tile
  static constexpr int NCH = 2;                           // chains
  static constexpr int WPC = 2;                           // warpgroups of math warps per chain, side by side
  static constexpr int CPT = BT / WPC;                    // columns of a tile per math thread
  static constexpr int NST = (DCH == 1) ? 5 : 4;          // ring of streamed tiles
  static constexpr int NB = (DCH == 1) ? 2 : 1;           // buffers for an item's own operands
  // dQ: dO rows for delta come from an item's own operand where its buffers are loaded early enough, O rows from memory
  static constexpr bool DO_SMEM = !DKV && NB > 1;
  static constexpr int NSB = 4;                           // dQ: items whose row statistics are at hand
  static constexpr int OP = DCH * 16384, HALF = DCH * BT * 128, STAGE = 2 * HALF;
  static constexpr int COL_D = BT, COLS = 2 * BT;         // TMEM columns of a chain: S at 0, dP at COL_D
  static constexpr int COL_B = NCH * COLS;                // dQ or dK
  static constexpr int NACC = DKV ? 1 : (512 - COL_B) / HD > 1 ? 2 : 1;     // accumulators of dQ, of dK
  static constexpr int COL_A = COL_B + HD;                // dV
  static constexpr int OUT_BYTES = 4 * 4096;              // two buffers of 32 rows x 32 columns per epilogue warp
  static constexpr int STAT = DKV ? NST * 2 * BT : NSB * 2 * TILE;
  static constexpr int SMEM = NB * 2 * OP + NST * STAGE + OUT_BYTES + STAT * 4 + 512;
  // warps: epilogue; math from 4 on; loads, the two issuers, one without work
  static constexpr int W_EPI = 0, W_MATH = 4, W_LOAD = 4 + 4 * NCH * WPC, W_A = W_LOAD + 1, W_B = W_LOAD + 2;
  static constexpr int THREADS = 32 * (W_LOAD + 4);
  // registers: together what 768 threads are launched with (80 each; checked before the launch)
  static constexpr int REGS_MATH = 88, REGS_REST = 64;
  static constexpr int REGS = 32 * (4 * NCH * WPC * REGS_MATH + 8 * REGS_REST);
  // where the bf16 pairs of columns 16 k .. 16 k + 15 lie: at the front of their warpgroup's columns
  static __host__ __device__ constexpr int word(int k) { return 16 * k / CPT * CPT + (16 * k % CPT) / 2; }
  static_assert(SMEM <= 227 * 1024, "shared memory");
  static_assert(COL_B + (DKV ? 2 : NACC) * HD <= 512, "TMEM columns");
  static_assert(CPT % 16 == 0, "products take 16 columns at a time");
};

struct BwdBars {
  uint64_t i0_full[2], i0_empty[2], i1_full[2], i1_empty[2];
  uint64_t r_full[5], r_empty[5];
  uint64_t s_full[2];       // scores of a tile are in the chain's TMEM columns
  uint64_t s_done[2];       // dQ: they have been read; dK/dV: P has taken their place
  uint64_t dp_full[2];      // dP is
  uint64_t ds_full[2];      // dS has taken its place
  uint64_t a_full, a_empty; // dV
  uint64_t b_full[2], b_empty[2];
  uint64_t stat_full[4], stat_empty[4];
};
static_assert(sizeof(BwdBars) + 8 + 4 * 4 <= 512, "barriers");

// Asynchronous 4-byte copy (`bytes` = 0: zero fill), and this lane's arrival on a barrier once its copies have landed.
__device__ __forceinline__ void cp_async4(float* smem_dst, const float* src, uint32_t bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(smem_dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Gradient rows on their way out: a warp turns 32 accumulator columns of its 32 rows into bf16 in shared memory, one lane
// hands them to the TMA unit as a tiled store. Rows past the window's end and columns past the head's width are clipped by
// the tensor map. No warp waits for another one's rows.
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

template <int DCH, bool DKV>
__global__ void __launch_bounds__(BwdCfg<DCH, DKV>::THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tm_i0, const __grid_constant__ CUtensorMap tm_i1,
                const __grid_constant__ CUtensorMap tm_r0, const __grid_constant__ CUtensorMap tm_r1,
                const __grid_constant__ CUtensorMap tm_out_b, const __grid_constant__ CUtensorMap tm_out_a,
                const AttnBwdParams p, const int n_items_total) {
  using R = BwdCfg<DCH, DKV>;
  constexpr int HD = R::HD, BT = R::BT, NCH = R::NCH, NST = R::NST, NB = R::NB, CPT = R::CPT;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* s_i0 = smem;                          // [NB]
  uint8_t* s_i1 = s_i0 + NB * R::OP;             // [NB]
  uint8_t* s_r = s_i1 + NB * R::OP;              // [NST] R0 | R1
  uint8_t* s_out = s_r + NST * R::STAGE;
  // dQ: [NSB] items: lse [128] | delta [128]; dK/dV: [NST] tiles: lse [BT] | delta [BT]
  float* s_stat = reinterpret_cast<float*>(s_out + R::OUT_BYTES);
  BwdBars* bar = reinterpret_cast<BwdBars*>(s_stat + R::STAT);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
  int* s_failed = s_abort + 1;      // [4] see note_failure

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int N = p.N;
  const int nfull = N / BT, rem = N - nfull * BT;
  const int n_str = nfull + (rem ? 1 : 0);                // streamed tiles of an item
  const int n_last = rem ? ((rem + 15) & ~15) : BT;       // columns of the products with the last one
  const int row_tiles = (N + TILE - 1) / TILE;
  const int n_ctas = static_cast<int>(gridDim.x);
  const int n_items = (n_items_total - static_cast<int>(blockIdx.x) + n_ctas - 1) / n_ctas;
  const int total = n_items * n_str;

  if (threadIdx.x == 0) {
    int ab = (p.status && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
    if ((smem_u32(smem) & 1023u) != 0) { ab = 1; if (p.status) atomicCAS(p.status, 0, ERR_BOUNDS); }
    *s_abort = ab;
  }
  __syncthreads();
  if (*s_abort) { chain_point(); return; }
  if (threadIdx.x == 0) {
    prefetch_tmap(&tm_i0); prefetch_tmap(&tm_i1); prefetch_tmap(&tm_r0); prefetch_tmap(&tm_r1);
    for (int i = 0; i < NB; ++i) {
      mbar_init(&bar->i0_full[i], 1); mbar_init(&bar->i0_empty[i], 1);
      mbar_init(&bar->i1_full[i], 1); mbar_init(&bar->i1_empty[i], R::DO_SMEM ? 1 + 4 : 1);
    }
    // a streamed tile's arrivals: the TMA loads and, for dK/dV, 32 lanes of row statistics. It is free after its last use by
    // either issuer: dQ's only one (dS K) comes last, dV and dK are issued by one each.
    for (int i = 0; i < NST; ++i) { mbar_init(&bar->r_full[i], DKV ? 1 + 32 : 1); mbar_init(&bar->r_empty[i], DKV ? 2 : 1); }
    for (int i = 0; i < NCH; ++i) {
      mbar_init(&bar->s_full[i], 1); mbar_init(&bar->s_done[i], 4 * R::WPC);
      mbar_init(&bar->dp_full[i], 1); mbar_init(&bar->ds_full[i], 4 * R::WPC);
    }
    mbar_init(&bar->a_full, 1); mbar_init(&bar->a_empty, 4);
    for (int i = 0; i < R::NACC; ++i) { mbar_init(&bar->b_full[i], 1); mbar_init(&bar->b_empty[i], 4); }
    for (int i = 0; i < R::NSB; ++i) { mbar_init(&bar->stat_full[i], 4); mbar_init(&bar->stat_empty[i], 4 * NCH * R::WPC); }
    fence_barrier_init();
  }
  if (warp == R::W_A) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_point();

  if ((warp & ~3) == R::W_LOAD) {
    regs_dec<R::REGS_REST>();
    if (warp == R::W_LOAD) {
      // ---------------------------------------------------------- TMA producer, one lane; dK/dV: all lanes copy statistics
      // (asynchronous 4-byte copies: a window's first row need not be 16-byte aligned; rows past its end become zeros).
      // The warp decides as one, so that its lanes stay together.
      auto wait = [&](uint64_t* b, uint32_t ph) -> bool {
        return mbar_wait_warp(b, ph, p.status, ERR_TIMEOUT_ATTN);
      };
      Slot is;
      auto load_item = [&](int it) -> bool {
        const BwdItem w = bwd_item(it, row_tiles, p.H);
        if (!wait(&bar->i0_empty[is.i], is.ph ^ 1)) return false;
        if (lane == 0) {
          mbar_expect_tx(&bar->i0_full[is.i], R::OP);
#pragma unroll
          for (int c = 0; c < DCH; ++c)
            tma_load_4d(s_i0 + is.i * R::OP + c * 16384, &tm_i0, &bar->i0_full[is.i], c * 64, w.head, w.tile * TILE, w.win);
        }
        if (!wait(&bar->i1_empty[is.i], is.ph ^ 1)) return false;
        if (lane == 0) {
          mbar_expect_tx(&bar->i1_full[is.i], R::OP);
#pragma unroll
          for (int c = 0; c < DCH; ++c)
            tma_load_4d(s_i1 + is.i * R::OP + c * 16384, &tm_i1, &bar->i1_full[is.i], c * 64, w.head, w.tile * TILE, w.win);
        }
        is.next(NB);
        return true;
      };
      // Where an item's own operands are requested: with several buffers those of the item NB - 1 on early in this one, with
      // one buffer those of this item behind its first tiles (they have to wait for the last products of the item before).
      constexpr int AHEAD = NB - 1;
      bool ok = true;
      for (int i = 0; i < (AHEAD ? AHEAD : 1) && i < n_items && ok; ++i) ok = load_item(i);
      const int j_item = min(AHEAD ? 2 : NCH - 1, n_str - 1);
      Slot rs;
      for (int it = 0; it < n_items && ok; ++it) {
        const BwdItem w = bwd_item(it, row_tiles, p.H);
        const size_t sbase = (static_cast<size_t>(w.win) * p.H + w.head) * N;
        for (int j = 0; j < n_str; ++j) {
          if (!wait(&bar->r_empty[rs.i], rs.ph ^ 1)) { ok = false; break; }
          uint64_t* full = &bar->r_full[rs.i];
          if (lane == 0) {
            uint8_t* d = s_r + rs.i * R::STAGE;
            mbar_expect_tx(full, R::STAGE);
#pragma unroll
            for (int c = 0; c < DCH; ++c) {
              tma_load_4d(d + c * (BT * 128), &tm_r0, full, c * 64, w.head, j * BT, w.win);
              tma_load_4d(d + R::HALF + c * (BT * 128), &tm_r1, full, c * 64, w.head, j * BT, w.win);
            }
          }
          if constexpr (DKV) {
            float* d = s_stat + rs.i * 2 * BT + lane;
#pragma unroll
            for (int u = 0; u < BT / 32; ++u) {
              const int r = j * BT + u * 32 + lane;
              const uint32_t bytes = (r < N) ? 4u : 0u;
              const size_t src = sbase + (r < N ? r : 0);
              cp_async4(d + u * 32, p.lse + src, bytes);
              cp_async4(d + BT + u * 32, p.delta + src, bytes);
            }
            cp_async_arrive(full);
          }
          rs.next(NST);
          if (j == j_item) {
            const int nxt = AHEAD ? it + AHEAD : it;
            if (nxt < n_items && (AHEAD || it > 0) && !load_item(nxt)) { ok = false; break; }
          }
        }
      }
      if constexpr (DKV) asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == R::W_A) {
      // ------------------------------------------------------------ issuer of the scores and, for dK/dV, of dV
      {
        const uint32_t lead = elect_one_sync();
        constexpr uint32_t idesc_acc = make_idesc_bf16(TILE, HD, 0, 1), idesc_full = make_idesc_bf16(TILE, BT, 0, 0);
        const uint32_t idesc_last = make_idesc_bf16(TILE, n_last, 0, 0);
        const uint32_t b_r = smem_u32(bar->r_full), b_s = smem_u32(bar->s_full), b_i = smem_u32(bar->i0_full);
        constexpr uint32_t B_REMPTY = offsetof(BwdBars, r_empty) - offsetof(BwdBars, r_full),
                           B_DONE = offsetof(BwdBars, s_done) - offsetof(BwdBars, s_full),
                           B_IEMPTY = offsetof(BwdBars, i0_empty) - offsetof(BwdBars, i0_full);
        const uint32_t lo_i = smem_desc_lo(smem_u32(s_i0), 0), lo_r = smem_desc_lo(smem_u32(s_r), 0);
        const uint32_t lo_a = smem_desc_lo(smem_u32(s_r) + R::HALF, BT * 128);
        Slot sw, ss, si;                  // chain, ring slot and item buffer of the tile whose scores are issued
        int j = 0, aj = 0, as = 0;        // its place in its item; place and ring slot of the tile NCH before it
        uint32_t a_ph = 1;                // of the accumulator: nothing to wait for the first time
        uint32_t w_ph = 0;                // of that tile in its chain
        auto scores = [&]() -> bool {
          if (j == 0 && !mbar_wait_warp(b_i + si.i * 8, si.ph, p.status, ERR_TIMEOUT_ATTN)) return false;
          tc_fence_after();
          const bool last = j == n_str - 1;
          const uint32_t idesc = last ? idesc_last : idesc_full, lo = lo_i + si.i * (R::OP / 16);
          const uint32_t tS = tmem_base + sw.i * R::COLS, lo_t = lo_r + ss.i * (R::STAGE / 16);
#pragma unroll
          for (int kk = 0; kk < 4 * DCH; ++kk)
            umma_ss_warp(lead, tS, smem_desc(lo + ((kk >> 2) * 16384 + (kk & 3) * 32) / 16),
                         smem_desc(lo_t + ((kk >> 2) * (BT * 128) + (kk & 3) * 32) / 16), idesc, kk > 0);
          tc_commit_warp(lead, b_s + sw.i * 8);
          ++j;
          if (last) { tc_commit_warp(lead, b_i + B_IEMPTY + si.i * 8); si.next(NB); j = 0; }
          ss.next(NST);
          return true;
        };
        // The tile NCH before it, whose columns the scores take: its own have been read (dQ), or turned into P, which
        // dV += P^T dO takes (A from TMEM, 16 columns = 8 words per K step; B MN-major: d contiguous).
        auto previous = [&]() -> bool {
          if constexpr (DKV) {
            if (aj == 0) {
              if (!mbar_wait_warp(smem_u32(&bar->a_empty), a_ph, p.status, ERR_TIMEOUT_ATTN)) return false;
              a_ph ^= 1;
            }
            tc_fence_after();
            const bool last = aj == n_str - 1;
            const uint32_t acc0 = aj > 0 ? 1u : 0u, tA = tmem_base + sw.i * R::COLS, tAcc = tmem_base + R::COL_A;
            const uint32_t lo = lo_a + as * (R::STAGE / 16);
            const int cols = last ? n_last : BT;
#pragma unroll
            for (int kk = 0; kk < BT / 16; ++kk)
              if (kk * 16 < cols)
                umma_ts_warp(lead, tAcc, tA + R::word(kk), smem_desc(lo + kk * 128), idesc_acc, kk ? 1u : acc0);
            tc_commit_warp(lead, b_r + B_REMPTY + as * 8);
            ++aj;
            if (last) { tc_commit_warp(lead, smem_u32(&bar->a_full)); aj = 0; }
            if (++as == NST) as = 0;
          }
          w_ph ^= sw.i == NCH - 1;
          return true;
        };
        bool ok = true;
        int g = 0;
        for (; g < NCH && g < total && ok; ++g, sw.next(NCH))
          ok = mbar_wait_warp(b_r + ss.i * 8, ss.ph, p.status, ERR_TIMEOUT_ATTN) && scores();
        for (; g < total && ok; ++g) {
          ok = mbar_wait_warp(b_r + ss.i * 8, ss.ph, b_s + B_DONE + sw.i * 8, w_ph, p.status, ERR_TIMEOUT_ATTN);
          ok = ok && previous() && scores();
          sw.next(NCH);
        }
        if constexpr (DKV) {
          if (total < NCH) sw = Slot{};
          for (int t = total < NCH ? 0 : total - NCH; t < total && ok; ++t, sw.next(NCH))
            ok = mbar_wait_warp(b_s + B_DONE + sw.i * 8, w_ph, p.status, ERR_TIMEOUT_ATTN) && previous();
        }
      }
    } else if (warp == R::W_B) {
      // ------------------------------------------------------------ issuer of dP and of dQ or dK
      {
        const uint32_t lead = elect_one_sync();
        constexpr uint32_t idesc_acc = make_idesc_bf16(TILE, HD, 0, 1), idesc_full = make_idesc_bf16(TILE, BT, 0, 0);
        const uint32_t idesc_last = make_idesc_bf16(TILE, n_last, 0, 0);
        const uint32_t b_r = smem_u32(bar->r_full), b_d = smem_u32(bar->dp_full), b_i = smem_u32(bar->i1_full),
                       b_b = smem_u32(bar->b_full);
        constexpr uint32_t B_REMPTY = offsetof(BwdBars, r_empty) - offsetof(BwdBars, r_full),
                           B_DONE = offsetof(BwdBars, ds_full) - offsetof(BwdBars, dp_full),
                           B_IEMPTY = offsetof(BwdBars, i1_empty) - offsetof(BwdBars, i1_full),
                           B_BEMPTY = offsetof(BwdBars, b_empty) - offsetof(BwdBars, b_full);
        const uint32_t lo_i = smem_desc_lo(smem_u32(s_i1), 0), lo_r = smem_desc_lo(smem_u32(s_r) + R::HALF, 0);
        const uint32_t lo_a = smem_desc_lo(smem_u32(s_r), BT * 128);
        Slot sw, ss, si, ac;              // chain, ring slot and item buffer of the tile whose dP is issued; accumulator
        int j = 0, aj = 0, as = 0;
        uint32_t w_ph = 0;
        auto issue_dp = [&]() -> bool {
          if (j == 0 && !mbar_wait_warp(b_i + si.i * 8, si.ph, p.status, ERR_TIMEOUT_ATTN)) return false;
          tc_fence_after();
          const bool last = j == n_str - 1;
          const uint32_t idesc = last ? idesc_last : idesc_full, lo = lo_i + si.i * (R::OP / 16);
          const uint32_t tD = tmem_base + sw.i * R::COLS + R::COL_D, lo_t = lo_r + ss.i * (R::STAGE / 16);
#pragma unroll
          for (int kk = 0; kk < 4 * DCH; ++kk)
            umma_ss_warp(lead, tD, smem_desc(lo + ((kk >> 2) * 16384 + (kk & 3) * 32) / 16),
                         smem_desc(lo_t + ((kk >> 2) * (BT * 128) + (kk & 3) * 32) / 16), idesc, kk > 0);
          tc_commit_warp(lead, b_d + sw.i * 8);
          ++j;
          if (last) { tc_commit_warp(lead, b_i + B_IEMPTY + si.i * 8); si.next(NB); j = 0; }
          ss.next(NST);
          return true;
        };
        auto accumulate = [&]() -> bool {
          if (aj == 0 && !mbar_wait_warp(b_b + B_BEMPTY + ac.i * 8, ac.ph ^ 1, p.status, ERR_TIMEOUT_ATTN)) return false;
          tc_fence_after();
          const bool last = aj == n_str - 1;
          const uint32_t acc0 = aj > 0 ? 1u : 0u, tA = tmem_base + sw.i * R::COLS + R::COL_D;
          const uint32_t tAcc = tmem_base + R::COL_B + ac.i * HD, lo = lo_a + as * (R::STAGE / 16);
          const int cols = last ? n_last : BT;
#pragma unroll
          for (int kk = 0; kk < BT / 16; ++kk)
            if (kk * 16 < cols)
              umma_ts_warp(lead, tAcc, tA + R::word(kk), smem_desc(lo + kk * 128), idesc_acc, kk ? 1u : acc0);
          tc_commit_warp(lead, b_r + B_REMPTY + as * 8);
          ++aj;
          if (last) { tc_commit_warp(lead, b_b + ac.i * 8); ac.next(R::NACC); aj = 0; }
          if (++as == NST) as = 0;
          w_ph ^= sw.i == NCH - 1;
          return true;
        };
        bool ok = true;
        int g = 0;
        for (; g < NCH && g < total && ok; ++g, sw.next(NCH))
          ok = mbar_wait_warp(b_r + ss.i * 8, ss.ph, p.status, ERR_TIMEOUT_ATTN) && issue_dp();
        for (; g < total && ok; ++g) {
          ok = mbar_wait_warp(b_r + ss.i * 8, ss.ph, b_d + B_DONE + sw.i * 8, w_ph, p.status, ERR_TIMEOUT_ATTN);
          // the tensor core executes in issue order: dP overwrites the A operand of the products before it after they have
          ok = ok && accumulate() && issue_dp();
          sw.next(NCH);
        }
        if (total < NCH) sw = Slot{};
        for (int t = total < NCH ? 0 : total - NCH; t < total && ok; ++t, sw.next(NCH))
          ok = mbar_wait_warp(b_d + B_DONE + sw.i * 8, w_ph, p.status, ERR_TIMEOUT_ATTN) && accumulate();
      }
    }
  } else if ((warp & ~3) == R::W_EPI) {
    regs_dec<R::REGS_REST>();
    // ------------------------------------------------------------ epilogue; dQ: also lse and delta of the coming items
    const int q = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    note_failure(p.status, &s_failed[q]);
    __syncwarp();
    BwdOut out{s_out + q * 4096, lane, q * 32};
    Slot sb, si;
    auto statistics = [&](int it) -> bool {
      constexpr int LPR = HD / 8, RPW = 32 / LPR;      // lanes per row, rows per load of this warp
      constexpr int UN = R::DO_SMEM ? 8 : 2;           // loads in flight
      const int sub = lane % LPR, r0 = lane / LPR;
      if (!mbar_wait_warp(&bar->stat_empty[sb.i], sb.ph ^ 1, p.status, ERR_TIMEOUT_ATTN)) return false;
      const BwdItem w = bwd_item(it, row_tiles, p.H);
      float* st = s_stat + sb.i * 2 * TILE;
      const size_t sbase = (static_cast<size_t>(w.win) * p.H + w.head) * N + w.tile * TILE;
      const int live = N - w.tile * TILE;            // rows of this tile inside the window
      const float lse = (q * 32 + lane < live) ? p.lse[sbase + q * 32 + lane] : 0.f;
      const size_t o0 = (static_cast<size_t>(w.win) * N + w.tile * TILE + q * 32 + r0) * p.ldo + w.head * p.d + sub * 8;
      const __nv_bfloat16 *po = p.O + o0, *pg = p.dO + o0;
      const int step = RPW * p.ldo;
#pragma unroll 1
      for (int r = q * 32; r < q * 32 + 32; r += RPW * UN) {
        uint4 a[UN], g[R::DO_SMEM ? 1 : UN];
#pragma unroll
        for (int u = 0; u < UN; ++u) {
          const bool in = r + u * RPW + r0 < live && sub * 8 < p.d;
          a[u] = in ? *reinterpret_cast<const uint4*>(po) : make_uint4(0u, 0u, 0u, 0u);
          po += step;
          if constexpr (!R::DO_SMEM) {
            g[u] = in ? *reinterpret_cast<const uint4*>(pg) : make_uint4(0u, 0u, 0u, 0u);
            pg += step;
          }
        }
        if constexpr (R::DO_SMEM)
          if (r == q * 32 && !mbar_wait_warp(&bar->i1_full[si.i], si.ph, p.status, ERR_TIMEOUT_ATTN)) return false;
#pragma unroll
        for (int u = 0; u < UN; ++u) {
          const int row = r + u * RPW + r0;
          uint4 y;
          if constexpr (R::DO_SMEM)
            y = *reinterpret_cast<const uint4*>(s_i1 + si.i * R::OP + (sub >> 3) * 16384 + swz128(row, sub & 7));
          else
            y = g[u];
          const uint32_t x4[4] = {a[u].x, a[u].y, a[u].z, a[u].w}, y4[4] = {y.x, y.y, y.z, y.w};
          float d = 0.f;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 x = unpack_bf16x2(x4[i]), z = unpack_bf16x2(y4[i]);
            d = fmaf(x.x, z.x, d);
            d = fmaf(x.y, z.y, d);
          }
#pragma unroll
          for (int o = LPR / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
          if (sub == 0) {
            st[TILE + row] = d;
            if (row < live) p.delta[sbase + row] = d;
          }
        }
      }
      if constexpr (R::DO_SMEM) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar->i1_empty[si.i]);
        si.next(NB);
      }
      st[q * 32 + lane] = lse;
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar->stat_full[sb.i]);
      sb.next(R::NSB);
      return true;
    };
    // HD accumulator columns at `t` of item `w` to memory; `empty` is told once they have been read
    auto drain = [&](uint32_t t, float f, const CUtensorMap* m, int section, int col0, const BwdItem& w, uint64_t* empty) {
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(empty);
      };
      const int n = (p.d + 31) / 32, N_out = noted(&s_failed[q]) ? 0 : N;      // rows that leave
      if (p.push_n_local == 0) {
        for (int c = 0; c < n; ++c)
          out.put(t + lane_addr + c * 32, f, m, c * 32, w.head, w.tile * TILE, w.win, N_out,
                  [&] { if (c == n - 1) release(); });
        return;
      }
      const int grow = w.tile * TILE + q * 32 + lane;
      const bool row_ok = grow < N_out;
      __nv_bfloat16* dst = bwd_dst(p, w.win, row_ok ? grow : 0, w.head, section, col0);
      for (int c = 0; c < n; ++c) {
        uint32_t v[32];
        tmem_ld32(t + lane_addr + c * 32, v);
        tmem_wait_ld();
        if (c == n - 1) release();
        if (row_ok) {
#pragma unroll
          for (int gq = 0; gq < 4; ++gq) {
            uint32_t o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              o[i] = pack_bf16x2(__uint_as_float(v[8 * gq + 2 * i]) * f, __uint_as_float(v[8 * gq + 2 * i + 1]) * f);
            if (c * 32 + gq * 8 < p.d)
              *reinterpret_cast<uint4*>(dst + c * 32 + gq * 8) = make_uint4(o[0], o[1], o[2], o[3]);
          }
        }
        __syncwarp();
      }
    };
    // O and dO rows of an item on their way to L2 (short windows: 200 x 225, 12 x 128 0.532 -> 0.478 ms)
    auto prefetch = [&](int it) {
      const BwdItem w = bwd_item(it, row_tiles, p.H);
      const int r = w.tile * TILE + q * 32 + lane;
      if (r < N) {
        const size_t o = (static_cast<size_t>(w.win) * N + r) * p.ldo + w.head * p.d;
        for (int c = 0; c < p.d; c += 64) {
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p.O + o + c));
          asm volatile("prefetch.global.L2 [%0];" ::"l"(p.dO + o + c));
        }
      }
      __syncwarp();
    };
    constexpr int AHEAD = R::DO_SMEM ? 1 : 2;      // items
    bool ok = true;
    if constexpr (!DKV)
      for (int i = 0; i < AHEAD && i < n_items && ok; ++i) ok = statistics(i);
    Slot ac;
    for (int it = 0; it < n_items && ok; ++it) {
      if constexpr (!DKV && !R::DO_SMEM)
        if (it + AHEAD + 1 < n_items) prefetch(it + AHEAD + 1);
      if constexpr (!DKV)
        if (it + AHEAD < n_items && !statistics(it + AHEAD)) { ok = false; break; }
      const BwdItem w = bwd_item(it, row_tiles, p.H);
      if constexpr (DKV) {
        if (!mbar_wait_warp(&bar->a_full, it & 1, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
        tc_fence_after();
        drain(tmem_base + R::COL_A, 1.f, &tm_out_a, 2, p.v_col0, w, &bar->a_empty);
      }
      if (!mbar_wait_warp(&bar->b_full[ac.i], ac.ph, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
      tc_fence_after();
      drain(tmem_base + R::COL_B + ac.i * HD, p.scale, &tm_out_b, DKV ? 1 : 0, DKV ? p.k_col0 : p.q_col0, w,
            &bar->b_empty[ac.i]);
      ac.next(R::NACC);
    }
    out.drain();
  } else {
    // ---------------------------------------------------------- math: one thread = CPT columns of a row, every NCH-th tile
    regs_inc<R::REGS_MATH>();
    const int wg = (warp >> 2) - 1, q = warp & 3;
    const int ch = wg / R::WPC, c0 = (wg % R::WPC) * CPT;           // chain, first column
    const int row = q * 32 + lane;
    const uint32_t tS = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + ch * R::COLS + c0, tD = tS + R::COL_D;
    uint32_t ph = 0;
    int j = ch;                       // first tile of this chain in the item at hand
    bool ok = true;
    auto wait = [&](uint64_t* b, uint32_t parity) -> bool {
      if (!mbar_wait_warp(b, parity, p.status, ERR_TIMEOUT_ATTN)) return false;
      tc_fence_after();
      return true;
    };
    auto tell = [&](uint64_t* b) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(b);
    };
    // CPT columns to registers
    auto load = [&](uint32_t t, uint32_t (&v)[CPT]) {
#pragma unroll
      for (int c = 0; c < CPT; c += 16) tmem_ld16(t + c, *reinterpret_cast<uint32_t(*)[16]>(&v[c]));
      tmem_wait_ld();
    };
    if constexpr (!DKV) {
      const uint64_t sl = f2_pack(p.scale_log2, p.scale_log2);
      Slot sb;
      for (int it = 0; it < n_items && ok; ++it) {
        if (!mbar_wait_warp(&bar->stat_full[sb.i], sb.ph, p.status, ERR_TIMEOUT_ATTN)) { ok = false; break; }
        const float nlse = -s_stat[sb.i * 2 * TILE + row], ndelta = -s_stat[sb.i * 2 * TILE + TILE + row];
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar->stat_empty[sb.i]);
        sb.next(R::NSB);
        const uint64_t nl = f2_pack(nlse, nlse), nd = f2_pack(ndelta, ndelta);
        for (; j < n_str; j += NCH, ph ^= 1) {
          if (!wait(&bar->s_full[ch], ph)) { ok = false; break; }
          if (j < nfull) {
            uint32_t pr[CPT];
            load(tS, pr);
            tell(&bar->s_done[ch]);
#pragma unroll
            for (int i = 0; i < CPT; i += 2) {
              float t0, t1;
              f2_unpack(f2_fma(f2_pack(__uint_as_float(pr[i]), __uint_as_float(pr[i + 1])), sl, nl), t0, t1);
              pr[i] = __float_as_uint(fast_exp2(t0));           // in place: ahead of the wait
              pr[i + 1] = __float_as_uint(fast_exp2(t1));
            }
            if (!wait(&bar->dp_full[ch], ph)) { ok = false; break; }
#pragma unroll
            for (int c = 0; c < CPT; c += 16) {
              uint32_t dv[16], pk[8];
              tmem_ld16(tD + c, dv);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const uint64_t df = f2_add(f2_pack(__uint_as_float(dv[2 * i]), __uint_as_float(dv[2 * i + 1])), nd);
                const uint64_t p2 = f2_pack(__uint_as_float(pr[c + 2 * i]), __uint_as_float(pr[c + 2 * i + 1]));
                pk[i] = f2_to_bf16x2(f2_mul(p2, df));
              }
              // 16 columns become 8 words at column c / 2 <= c: only columns that were read are overwritten
              tmem_st8(tD + (c >> 1), pk);
            }
          } else {
            // columns past the window's end: their K rows are zeros, but an exponential may be infinite there
            if (!wait(&bar->dp_full[ch], ph)) { ok = false; break; }
#pragma unroll 1
            for (int c = 0; c < CPT && c0 + c < n_last; c += 16) {
              uint32_t sv[16], dv[16], pk[8];
              tmem_ld16(tS + c, sv);
              tmem_ld16(tD + c, dv);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const float p0 = mufu_exp2(fmaf(__uint_as_float(sv[2 * i]), p.scale_log2, nlse));
                const float p1 = mufu_exp2(fmaf(__uint_as_float(sv[2 * i + 1]), p.scale_log2, nlse));
                float d0 = p0 * (__uint_as_float(dv[2 * i]) + ndelta);
                float d1 = p1 * (__uint_as_float(dv[2 * i + 1]) + ndelta);
                if (c0 + c + 2 * i >= rem) d0 = 0.f;
                if (c0 + c + 2 * i + 1 >= rem) d1 = 0.f;
                pk[i] = pack_bf16x2(d0, d1);
              }
              tmem_st8(tD + (c >> 1), pk);
            }
            tell(&bar->s_done[ch]);
          }
          tmem_wait_st();
          tell(&bar->ds_full[ch]);
        }
        j -= n_str;                      // the stream of tiles runs on into the next item
      }
    } else {
      const uint64_t nsl = f2_pack(-p.scale_log2, -p.scale_log2);
      // Columns past the window's end have zero Q and dO rows and zero statistics (P = 1, dS = 0): they add nothing. Rows
      // past its end may hold anything: they are not stored.
      auto probs = [&](uint32_t& s0, uint32_t& s1, uint64_t l) -> uint32_t {
        float t0, t1;
        f2_unpack(f2_fma(f2_pack(__uint_as_float(s0), __uint_as_float(s1)), nsl, l), t0, t1);     // -(log2 P)
        t0 = fast_exp2(-t0);
        t1 = fast_exp2(-t1);
        s0 = __float_as_uint(t0);
        s1 = __float_as_uint(t1);
        return pack_bf16x2(t0, t1);
      };
      auto grad = [&](uint32_t p0, uint32_t p1, uint32_t d0, uint32_t d1, uint64_t de) -> uint32_t {
        return f2_to_bf16x2(f2_mul(f2_pack(__uint_as_float(p0), __uint_as_float(p1)),
                                   f2_sub(f2_pack(__uint_as_float(d0), __uint_as_float(d1)), de)));
      };
      int st = ch;
      for (int it = 0; it < n_items && ok; ++it) {
        for (; j < n_str; j += NCH, ph ^= 1, st = st + NCH >= NST ? st + NCH - NST : st + NCH) {
          if (!wait(&bar->s_full[ch], ph)) { ok = false; break; }
          const ulonglong2* ls = reinterpret_cast<const ulonglong2*>(s_stat + st * 2 * BT + c0);
          const ulonglong2* ds = ls + BT / 4;
          if (j < nfull) {
            uint32_t pr[CPT];
            load(tS, pr);
#pragma unroll
            for (int c = 0; c < CPT; c += 16) {
              uint32_t pp[8];
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const ulonglong2 l = ls[c / 4 + i];
                pp[2 * i] = probs(pr[c + 4 * i], pr[c + 4 * i + 1], l.x);
                pp[2 * i + 1] = probs(pr[c + 4 * i + 2], pr[c + 4 * i + 3], l.y);
              }
              tmem_st8(tS + (c >> 1), pp);
            }
            tmem_wait_st();
            tell(&bar->s_done[ch]);
            if (!wait(&bar->dp_full[ch], ph)) { ok = false; break; }
#pragma unroll
            for (int c = 0; c < CPT; c += 16) {
              uint32_t dv[16], dd[8];
              tmem_ld16(tD + c, dv);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const ulonglong2 de = ds[c / 4 + i];
                dd[2 * i] = grad(pr[c + 4 * i], pr[c + 4 * i + 1], dv[4 * i], dv[4 * i + 1], de.x);
                dd[2 * i + 1] = grad(pr[c + 4 * i + 2], pr[c + 4 * i + 3], dv[4 * i + 2], dv[4 * i + 3], de.y);
              }
              tmem_st8(tD + (c >> 1), dd);
            }
          } else {
            if (!wait(&bar->dp_full[ch], ph)) { ok = false; break; }
#pragma unroll 1
            for (int c = 0; c < CPT && c0 + c < n_last; c += 16) {
              uint32_t sv[16], dv[16], pp[8], dd[8];
              tmem_ld16(tS + c, sv);
              tmem_ld16(tD + c, dv);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const ulonglong2 l = ls[c / 4 + i], de = ds[c / 4 + i];
                pp[2 * i] = probs(sv[4 * i], sv[4 * i + 1], l.x);
                pp[2 * i + 1] = probs(sv[4 * i + 2], sv[4 * i + 3], l.y);
                dd[2 * i] = grad(sv[4 * i], sv[4 * i + 1], dv[4 * i], dv[4 * i + 1], de.x);
                dd[2 * i + 1] = grad(sv[4 * i + 2], sv[4 * i + 3], dv[4 * i + 2], dv[4 * i + 3], de.y);
              }
              tmem_st8(tS + (c >> 1), pp);
              tmem_st8(tD + (c >> 1), dd);
            }
            tmem_wait_st();
            tell(&bar->s_done[ch]);
          }
          tmem_wait_st();
          tell(&bar->ds_full[ch]);
        }
        j -= n_str;                     // the stream of tiles runs on into the next item
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == R::W_A) tmem_dealloc(tmem_base, 512);
}

template <int DCH>
static int launch_attn_bwd(const CUtensorMap& tq128, const CUtensorMap& tk64, const CUtensorMap& tv64,
                           const CUtensorMap& tdo128, const CUtensorMap& tq64, const CUtensorMap& tk128,
                           const CUtensorMap& tv128, const CUtensorMap& tdo64, const CUtensorMap (&out)[3],
                           const AttnBwdParams& p, cudaStream_t stream) {
  using R1 = BwdCfg<DCH, false>;
  using R2 = BwdCfg<DCH, true>;
  auto k1 = attn_bwd_kernel<DCH, false>;
  auto k2 = attn_bwd_kernel<DCH, true>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, R1::SMEM) != cudaSuccess) return -20;
    if (cudaFuncSetAttribute(k2, cudaFuncAttributeMaxDynamicSharedMemorySize, R2::SMEM) != cudaSuccess) return -20;
    // warpgroups that ask for more registers than the launch holds would wait for ever
    cudaFuncAttributes f1, f2;
    if (cudaFuncGetAttributes(&f1, k1) != cudaSuccess || cudaFuncGetAttributes(&f2, k2) != cudaSuccess) return -20;
    if (f1.numRegs * R1::THREADS < R1::REGS || f2.numRegs * R2::THREADS < R2::REGS) return -24;
    configured = true;
  }
  const int n = (p.N + TILE - 1) / TILE * p.H * p.n_win, grid = n < num_sms() ? n : num_sms();
  if (launch_chained(k1, grid, R1::THREADS, R1::SMEM, stream, tq128, tdo128, tk64, tv64, out[0], out[0], p, n)) return -21;
  return launch_chained(k2, grid, R2::THREADS, R2::SMEM, stream, tk128, tv128, tq64, tdo64, out[1], out[2], p, n) ? -22 : 0;
}

}  // namespace aeris
