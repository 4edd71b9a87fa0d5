// Attention forward for heads up to 64 and windows of several query tiles: one persistent CTA per SM, four query tiles of
// 128 rows at a time (four "chains"), the window's K and V streamed once for all of them in tiles of 64 rows. Included
// by attention.cu.
//
// A chain is one after the other: products, maximum, exponentials, hand-over, products; two chains per SM
// (attention_fwd_pair.cuh) leave the exponential unit idle for 43 % of the time. Here four warps share a scheduler's, a
// chain's P lies over its scores in tensor memory (128 columns a chain, 64 of them O), and its next scores follow P V in
// issue order. Two warps issue the products of two chains each. An item's output rows leave while the first products of
// the next are already done. Reference maximum, sums and results are those of attn_fwd_kernel in every bit.
// 72 windows x 900 tokens, 24 heads x 64, bursts: 0.623 -> 0.553 ms; 24 x 32 0.617 -> 0.537; others at the rule in
// attention.cu. A chain's round: 2,760 cycles for 64 columns, 740 of them from its hand-over to the next scores, 220 to
// read them, 250 for the maximum, 1,150 of exponentials (512 by themselves), 165 to write P and hand over. The
// exponential unit is at 66 % (ncu, 36 windows).
// Tried: four issuers, one a chain, 0.571; a chain's last warp issuing its products itself 0.687.
#pragma once
#include <stddef.h>

namespace aeris {

struct AttnQuad {
  static constexpr int NC = 4;                              // chains
  static constexpr int NBQ = 2;                             // buffers per chain for its query tile
  static constexpr int NST = 4;                             // ring of K | V tiles
  static constexpr int Q_BYTES = 16384, HALF = KVT * 128, STAGE = 2 * HALF;
  static constexpr int OUT_BYTES = 2048;                    // per softmax warp: 32 rows x 32 columns
  static constexpr int SMEM = NC * NBQ * Q_BYTES + NST * STAGE + 4 * NC * OUT_BYTES + 512;
  // tensor memory, per chain: scores, over them P, then O
  static constexpr int COLS = 128, COL_O = 64;
  // warps: softmax, four per chain; loads; an issuer for two chains each; one without work
  static constexpr int W_LOAD = 4 * NC, W_ISSUE = W_LOAD + 1;
  static constexpr int THREADS = 32 * (W_LOAD + 4);
  static constexpr int REGS_SOFTMAX = 104, REGS_REST = 64;
  static constexpr int REGS = 32 * (4 * NC * REGS_SOFTMAX + 4 * REGS_REST);
};
static_assert(AttnQuad::SMEM <= 227 * 1024, "shared memory");

struct QuadBars {
  uint64_t q_full[4][2], q_empty[4][2];
  uint64_t t_full[4], t_empty[4];       // K and V of a tile
  uint64_t s_full[4];                   // the chain's scores are in tensor memory
  uint64_t p_full[4];                   // its probabilities have taken their place
  uint64_t o_full[4];                   // the last P V of an item has completed
};
static_assert(sizeof(QuadBars) + 8 + 4 * 16 <= 512, "barriers");

__global__ void __launch_bounds__(AttnQuad::THREADS, 1)
attn_fwd_quad_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                     const AttnFwdParams p, const int n_items_total) {
  using R = AttnQuad;
  constexpr int NC = R::NC, NBQ = R::NBQ, NST = R::NST;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;                               // [chains][NBQ]
  uint8_t* sT = sQ + NC * NBQ * R::Q_BYTES;         // [NST] K | V
  uint8_t* sO = sT + NST * R::STAGE;                // [softmax warps]
  QuadBars* bar = reinterpret_cast<QuadBars*>(sO + 4 * NC * R::OUT_BYTES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar + 1);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
  int* s_failed = s_abort + 1;      // [16] see note_failure

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int N = p.N;
  const int nfull = N / KVT, rem = N - nfull * KVT;
  const int nkv = nfull + (rem ? 1 : 0);
  const int n_last = rem ? ((rem + 15) & ~15) : KVT;      // columns computed in the last tile
  // an item: up to four query tiles of one (window, head); see pair_item
  const int q_tiles = (N + TILE - 1) / TILE, n_groups = (q_tiles + NC - 1) / NC;
  const int n_ctas = static_cast<int>(gridDim.x);
  const int n_items = (n_items_total - static_cast<int>(blockIdx.x) + n_ctas - 1) / n_ctas;
  const int total = n_items * nkv;

  if (threadIdx.x == 0) {
    int ab = (p.status && *reinterpret_cast<volatile int*>(p.status) != 0) ? 1 : 0;
    if ((smem_u32(smem) & 1023u) != 0) { ab = 1; if (p.status) atomicCAS(p.status, 0, ERR_BOUNDS); }
    *s_abort = ab;
  }
  __syncthreads();
  if (*s_abort) { chain_point(); return; }
  if (threadIdx.x == 0) {
    prefetch_tmap(&tm_q); prefetch_tmap(&tm_k); prefetch_tmap(&tm_v);
    for (int c = 0; c < NC; ++c) {
      for (int b = 0; b < NBQ; ++b) { mbar_init(&bar->q_full[c][b], 1); mbar_init(&bar->q_empty[c][b], 1); }
      mbar_init(&bar->s_full[c], 1); mbar_init(&bar->p_full[c], 4); mbar_init(&bar->o_full[c], 1);
    }
    for (int i = 0; i < NST; ++i) { mbar_init(&bar->t_full[i], 1); mbar_init(&bar->t_empty[i], 2); }
    fence_barrier_init();
  }
  if (warp == R::W_LOAD) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_point();

  if (warp >= R::W_LOAD) {
    regs_dec<R::REGS_REST>();
    if (warp == R::W_LOAD) {
      // ---------------------------------------------------------- TMA producer
      Slot qs[NC];
      auto load_q = [&](int it) -> bool {
        const PairItem w = pair_item(it, n_groups, p.H);
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int qt = NC * w.pair + c;
          if (qt >= q_tiles) continue;
          if (!mbar_wait_warp(&bar->q_empty[c][qs[c].i], qs[c].ph ^ 1, p.status, ERR_TIMEOUT_ATTN)) return false;
          if (lane == 0) {
            uint64_t* full = &bar->q_full[c][qs[c].i];
            mbar_expect_tx(full, R::Q_BYTES);
            tma_load_4d(sQ + (c * NBQ + qs[c].i) * R::Q_BYTES, &tm_q, full, 0, w.head, qt * TILE, w.win);
          }
          qs[c].next(NBQ);
        }
        return true;
      };
      bool ok = load_q(0);
      Slot ts;
      for (int it = 0; it < n_items && ok; ++it) {
        const PairItem w = pair_item(it, n_groups, p.H);
        for (int j = 0; j < nkv && ok; ++j) {
          ok = mbar_wait_warp(&bar->t_empty[ts.i], ts.ph ^ 1, p.status, ERR_TIMEOUT_ATTN);
          if (ok && lane == 0) {
            uint64_t* full = &bar->t_full[ts.i];
            uint8_t* d = sT + ts.i * R::STAGE;
            mbar_expect_tx(full, R::STAGE);
            tma_load_4d(d, &tm_k, full, 0, w.head, j * KVT, w.win);
            tma_load_4d(d + R::HALF, &tm_v, full, 0, w.head, j * KVT, w.win);
          }
          ts.next(NST);
          // the query tiles of the next item, early in this one
          if (ok && j == min(2, nkv - 1) && it + 1 < n_items) ok = load_q(it + 1);
        }
      }
    } else if (warp < R::W_ISSUE + 2) {
      // ---------------------------------------------------------- issuer of two chains' products
      const uint32_t lead = elect_one_sync();
      const int c0 = 2 * (warp - R::W_ISSUE);
      constexpr uint32_t idesc_pv = make_idesc_bf16(TILE, 64, 0, 1), idesc_full = make_idesc_bf16(TILE, KVT, 0, 0);
      const uint32_t idesc_last = make_idesc_bf16(TILE, n_last, 0, 0);
      const uint32_t lo_q = smem_desc_lo(smem_u32(sQ), 0), lo_k = smem_desc_lo(smem_u32(sT), 0);
      const uint32_t lo_v = smem_desc_lo(smem_u32(sT) + R::HALF, 8192);
      const uint32_t b_t = smem_u32(bar->t_full), b_s = smem_u32(bar->s_full), b_p = smem_u32(bar->p_full),
                     b_q = smem_u32(bar->q_full);
      constexpr uint32_t B_TEMPTY = offsetof(QuadBars, t_empty) - offsetof(QuadBars, t_full),
                         B_QEMPTY = offsetof(QuadBars, q_empty) - offsetof(QuadBars, q_full),
                         B_OFULL = offsetof(QuadBars, o_full) - offsetof(QuadBars, s_full);
      auto chains = [&](int it) { return min(NC, q_tiles - NC * pair_item(it, n_groups, p.H).pair) - c0; };
      Slot qs[2];                       // query buffers of the two chains
      uint32_t p_ph[2] = {};
      // S = Q K^T of ring slot `slot` for chain u
      auto scores = [&](int u, int slot, bool first, bool last) -> bool {
        const int c = c0 + u;
        if (first && !mbar_wait_warp(b_q + (c * 2 + qs[u].i) * 8, qs[u].ph, p.status, ERR_TIMEOUT_ATTN)) return false;
        tc_fence_after();
        const uint32_t a = lo_q + (c * NBQ + qs[u].i) * (R::Q_BYTES / 16), b = lo_k + slot * (R::STAGE / 16);
        const uint32_t idesc = last ? idesc_last : idesc_full;
        umma_ss4_warp<2, 2>(lead, tmem_base + c * R::COLS, a, b, idesc, 0);
        tc_commit_warp(lead, b_s + c * 8);
        if (last) { tc_commit_warp(lead, b_q + B_QEMPTY + (c * 2 + qs[u].i) * 8); qs[u].next(NBQ); }
        return true;
      };
      // O += P V (A = P in tensor memory, 16 columns of bf16 = 8 words per K step; B = V MN-major)
      auto product = [&](int u, int slot, bool first, bool last) {
        const uint32_t tS = tmem_base + (c0 + u) * R::COLS, b = lo_v + slot * (R::STAGE / 16);
        tc_fence_after();
        if (!last || rem == 0) {
          umma_ts4_warp<8, 128>(lead, tS + R::COL_O, tS, b, idesc_pv, !first);
        } else {
#pragma unroll 1
          for (int kk = 0; kk < n_last / 16; ++kk)
            umma_ts_warp(lead, tS + R::COL_O, tS + kk * 8, smem_desc(b + kk * 128), idesc_pv, kk || !first);
        }
        if (last) tc_commit_warp(lead, b_s + B_OFULL + (c0 + u) * 8);
        p_ph[u] ^= 1;
      };
      int n_now = chains(0), n_next = n_now;
      bool ok = mbar_wait_warp(b_t, 0, p.status, ERR_TIMEOUT_ATTN);
#pragma unroll
      for (int u = 0; u < 2; ++u)
        if (u < n_now && ok) ok = scores(u, 0, true, nkv == 1);
      int it = 0, j = 0, slot = 0;
      Slot ns;                          // the next tile's slot
      ns.next(NST);
      for (int g = 0; g < total && ok; ++g) {
        // the tile after this one: of this item, or the first of the next
        const bool last = j == nkv - 1, more = g + 1 < total;
        const int nj = last ? 0 : j + 1;
        if (last && more) n_next = chains(it + 1);
        if (more) ok = mbar_wait_warp(b_t + ns.i * 8, ns.ph, p.status, ERR_TIMEOUT_ATTN);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (ok && u < n_now) {
            ok = mbar_wait_warp(b_p + (c0 + u) * 8, p_ph[u], p.status, ERR_TIMEOUT_ATTN);
            if (ok) product(u, slot, j == 0, last);
          }
          if (u == 1) tc_commit_warp(lead, b_t + B_TEMPTY + slot * 8);
          // the scores overwrite P, which the tensor core has consumed by then: it executes in issue order
          if (ok && more && u < n_next) ok = scores(u, ns.i, nj == 0, nj == nkv - 1);
        }
        slot = ns.i;
        ns.next(NST);
        j = nj;
        if (last) { ++it; n_now = n_next; }
      }
    }
  } else {
    // ------------------------------------------------------------ softmax: one thread = one query row of its chain
    regs_inc<R::REGS_SOFTMAX>();
    const int c = warp >> 2, q = warp & 3;
    note_failure(p.status, &s_failed[warp]);
    const uint32_t tS = tmem_base + c * R::COLS + (static_cast<uint32_t>(q * 32) << 16), tO = tS + R::COL_O;
    const float sl2 = p.scale_log2;
    const uint64_t sl = f2_pack(sl2, sl2);
    uint8_t* stage = sO + warp * R::OUT_BYTES;
    uint32_t s_ph = 0, o_ph = 0;
    bool ok = true;
    float m_ref = 0.f, l = 0.f;
    // Output rows and row statistics of an item, whose last P V has completed. A warp's rows leave as tiles of 32 columns
    // through shared memory.
    auto epilogue = [&](const PairItem& w) {
      const int tile_row = (NC * w.pair + c) * TILE + q * 32, grow = tile_row + lane;
      const float inv = 1.f / l;
      __nv_bfloat16* pdst = nullptr;
      if (p.push_n_local > 0 && grow < N) {
        const int owner = grow / p.push_n_local;
        pdst = reinterpret_cast<__nv_bfloat16*>(p.o_peers[owner]) +
               (static_cast<size_t>(w.win) * p.push_n_local + (grow - owner * p.push_n_local)) * p.push_ld +
               p.push_col0 + w.head * p.d;
      }
#pragma unroll 1
      for (int col = 0; col < p.d; col += 32) {
        uint32_t v[32];
        tmem_ld32(tO + col, v);
        tmem_wait_ld();
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            o[i] = pack_bf16x2(__uint_as_float(v[8 * g + 2 * i]) * inv, __uint_as_float(v[8 * g + 2 * i + 1]) * inv);
          const uint4 u = make_uint4(o[0], o[1], o[2], o[3]);
          *reinterpret_cast<uint4*>(stage + lane * 64 + ((g ^ ((lane >> 1) & 3)) << 4)) = u;
          if (pdst && col + 8 * g < p.d) *reinterpret_cast<uint4*>(pdst + col + 8 * g) = u;
        }
        fence_proxy_async_smem();
        __syncwarp();
        // columns past the head's width and rows past the window's end are clipped
        if (lane == 0 && p.O) tma_store_4d(&tm_o, stage, col, w.head, tile_row, w.win);
        __syncwarp();
      }
      if (p.lse && grow < N) p.lse[(static_cast<size_t>(w.win) * p.H + w.head) * N + grow] = m_ref + log2f(l);
      __syncwarp();
    };
    // The reference maximum is raised when a row's maximum grows by more than 2^8; these scores were issued behind the P V
    // of the tile before, so the accumulator is up to date.
    auto raise = [&](int j, float mx) {
      const float m_new = fmaxf(m_ref, mx * sl2);
      if (__any_sync(0xffffffffu, m_new - m_ref > RESCALE_LOG2)) {
        if (j > 0) {
          const float alpha = fast_exp2(m_ref - m_new);
          rescale_tmem_rows(tO, 64, alpha);
          l *= alpha;
        }
        m_ref = m_new;
      }
    };
    bool pending = false;               // `prev` has rows that are still in tensor memory
    PairItem prev{0, 0, 0};
    for (int it = 0; it < n_items && ok; ++it) {
      const PairItem w = pair_item(it, n_groups, p.H);
      const int qt = NC * w.pair + c;
      if (qt >= q_tiles) continue;
      const bool rows = qt * TILE + q * 32 < N;
      for (int j = 0; j < nkv; ++j) {
        ok = mbar_wait_warp(&bar->s_full[c], s_ph, p.status, ERR_TIMEOUT_ATTN);
        if (!ok) break;
        s_ph ^= 1;
        tc_fence_after();
        if (j == 0) {
          // these scores were issued behind the last P V of the item before: its rows leave now
          if (pending && !noted(&s_failed[warp])) epilogue(prev);
          pending = rows;
          prev = w;
          m_ref = -INFINITY;
          l = 0.f;
        }
        if (!rows) {
        } else if (j < nfull) {
          uint32_t v[2][32];
          tmem_ld32(tS, v[0]);
          tmem_ld32(tS + 32, v[1]);
          tmem_wait_ld();
          float mx[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) mx[k] = fmaxf(__uint_as_float(v[0][k]), __uint_as_float(v[1][k]));
#pragma unroll
          for (int i = 4; i < 32; i += 4) {
#pragma unroll
            for (int k = 0; k < 4; ++k) mx[k] = max3(mx[k], __uint_as_float(v[0][i + k]), __uint_as_float(v[1][i + k]));
          }
          raise(j, fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]));
          const uint64_t nm = f2_pack(-m_ref, -m_ref);
          HalfSum sum;
          softmax_chunk<false>(v[0], sl, nm, sum, tS);          // over columns that have been read
          softmax_chunk<false>(v[1], sl, nm, sum, tS + 16);
          l += sum.total(false);
          tmem_wait_st();
        } else {
          // last, partial tile: n_last columns computed, `rem` of them valid
          float mx = -INFINITY;
#pragma unroll 1
          for (int k = 0; k < n_last; k += 16) {
            uint32_t v[16];
            tmem_ld16(tS + k, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (k + i < rem) mx = fmaxf(mx, __uint_as_float(v[i]));
          }
          raise(j, mx);
          float rs = 0.f;
#pragma unroll 1
          for (int k = 0; k < n_last; k += 16) {
            uint32_t v[16], pk[8];
            tmem_ld16(tS + k, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              float p0 = fast_exp2(fmaf(__uint_as_float(v[2 * i]), sl2, -m_ref));
              float p1 = fast_exp2(fmaf(__uint_as_float(v[2 * i + 1]), sl2, -m_ref));
              if (k + 2 * i >= rem) p0 = 0.f;
              if (k + 2 * i + 1 >= rem) p1 = 0.f;
              rs += p0 + p1;
              pk[i] = pack_bf16x2(p0, p1);
            }
            tmem_st8(tS + (k >> 1), pk);      // over columns that have been read
          }
          l += rs;
          tmem_wait_st();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar->p_full[c]);
      }
      o_ph ^= 1;
    }
    if (ok && pending && mbar_wait_warp(&bar->o_full[c], o_ph ^ 1, p.status, ERR_TIMEOUT_ATTN) && !noted(&s_failed[warp])) {
      tc_fence_after();
      epilogue(prev);
    }
    // the copies have been performed before their shared memory goes
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == R::W_LOAD) tmem_dealloc(tmem_base, 512);
}

static int launch_attn_fwd_quad(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                                const CUtensorMap& to, const AttnFwdParams& p, cudaStream_t stream) {
  using R = AttnQuad;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(attn_fwd_quad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, R::SMEM) != cudaSuccess)
      return -20;
    // warpgroups that ask for more registers than the launch holds would wait for ever
    cudaFuncAttributes f;
    if (cudaFuncGetAttributes(&f, attn_fwd_quad_kernel) != cudaSuccess) return -20;
    if (f.numRegs * R::THREADS < R::REGS) return -24;
    configured = true;
  }
  const int groups = ((p.N + TILE - 1) / TILE + R::NC - 1) / R::NC;
  const long long items = static_cast<long long>(groups) * p.H * p.n_win;
  const int nkv = (p.N + KVT - 1) / KVT;
  if (items > 0x3fffffff || items * nkv > 0x3fffffffll * num_sms()) return -23;
  const int n = static_cast<int>(items), grid = n < num_sms() ? n : num_sms();
  return launch_chained(attn_fwd_quad_kernel, grid, R::THREADS, R::SMEM, stream, tq, tk, tv, to, p, n);
}

}  // namespace aeris
