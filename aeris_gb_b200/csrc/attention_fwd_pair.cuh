// Attention forward for windows of more than one query tile: one persistent CTA per SM, two query tiles of 128 rows at a
// time (two "chains"), the window's K and V streamed once for both in tiles of 128 rows. Included by attention.cu.
//
// The kernel in attention.cu (three CTAs per SM, 64-column tiles) pays six hand-shakes of 200-300 cycles between softmax
// warps and tensor core per 64 columns, passes P through shared memory, whose bandwidth its N = 64 products already use up,
// and loads K and V once per query tile. Here a hand-shake is paid per 128 columns, products are 128 wide, P stays in tensor
// memory and K and V serve two tiles. What bounds it now is latency again: with two warps per scheduler the exponentials
// of a tile (711 cycles by themselves) take 1,100-1,700, and waits, maximum and hand-over another 1,000.
// Tensor memory: per chain 128 score columns, O, and P. At head_dim 64 P has columns of its own, so that the next scores are
// computed under the softmax; at 128 it lies over the scores, whose successors then wait for P V, and the chains take turns.
// The output is that of attn_fwd_kernel in every bit (reference maximum and sums go by 64 columns as there) unless the
// second half of a tile raises the reference maximum. Against one tile at a time, in turn under the power cap, ms, windows
// x tokens, 24 heads x 64 / 12 x 128: 72 x 900 0.734 -> 0.662 / 0.565 -> 0.487; 253 x 256 0.308 -> 0.216 / 0.275 -> 0.166;
// 288 x 225 0.303 -> 0.258 / 0.284 -> 0.182; 502 x 129 0.367 -> 0.318 / 0.307 -> 0.216; 55 x 1024 0.646 -> 0.543 / 0.489 ->
// 0.396; 8 x 900, 4 x 64: 0.0247 -> 0.0218. Maximum and sum over whole tiles would save 1-2 %, and 5-10 % where CUT.
// Tried: one piece of straight code per full tile and a rolled loop for the last one (no gain at 900 tokens, 225: 0.168 ->
// 0.190); strict turns of the two chains at the exponentials (0.620 -> 0.677); one warp for the products of both chains is
// not needed: issuing a tile's twelve products and their commits takes 400 cycles of 3,000.
#pragma once

namespace aeris {

constexpr int KVP = 128;      // rows of a streamed K or V tile

template <int DCH> struct AttnPair {
  static constexpr int Q_BYTES = DCH * 16384, T_BYTES = DCH * 16384;      // a query tile; a K or V tile
  static constexpr int NBQ = DCH == 1 ? 2 : 1;                            // buffers per chain for its query tile
  static constexpr int NS = DCH == 1 ? 3 : 2;                             // depth of the K ring and of the V ring
  static constexpr int OUT_BYTES = 16384;                                 // staging of 64 output columns, 4 KB a warp
  static constexpr int SMEM = 2 * NBQ * Q_BYTES + 2 * NS * T_BYTES + 2 * OUT_BYTES + 512;
  static constexpr int THREADS = 384;
  // tensor memory columns of a chain (256 each): scores at 0, then
  static constexpr int COL_P = DCH == 1 ? 128 : 0;
  static constexpr int COL_O = DCH == 1 ? 192 : 128;
};
static_assert(AttnPair<1>::SMEM <= 227 * 1024 && AttnPair<2>::SMEM <= 227 * 1024, "shared memory");

struct PairItem {
  int pair, head, win;
};
// Item `it` of this CTA. Pairs of one (window, head) are neighbours, so the CTAs at work share K and V in L2; which of them
// a CTA gets is rotated from round to round, because the last pair of a window may have a single chain.
__device__ __forceinline__ PairItem pair_item(int it, int n_pairs, int H) {
  const int idx = blockIdx.x + it * gridDim.x;
  const int wh = idx / n_pairs;
  PairItem b;
  b.pair = (idx - wh * n_pairs + (wh * n_pairs) / static_cast<int>(gridDim.x)) % n_pairs;
  b.win = wh / H;
  b.head = wh - b.win * H;
  return b;
}

// Sum of 64 probabilities of a row in the order in which attn_fwd_kernel adds them up: four sums by column, or pair after
// pair in a half tile that the window's end cuts off.
struct HalfSum {
  uint64_t by_col[2] = {0ull, 0ull};       // bit pattern of (0.f, 0.f)
  float in_row = 0.f;

  __device__ __forceinline__ float total(bool cut) const {
    float s0, s1, s2, s3;
    f2_unpack(by_col[0], s0, s1);
    f2_unpack(by_col[1], s2, s3);
    return cut ? in_row : (s0 + s1) + (s2 + s3);
  }
};

// Probabilities of 32 scores of a row against the reference maximum: bf16 pairs into tensor memory, added to `sum`.
template <bool IN_ROW>
__device__ __forceinline__ void softmax_chunk(const uint32_t (&v)[32], uint64_t sl, uint64_t nm, HalfSum& sum, uint32_t tP) {
  uint32_t pk[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    float t0, t1;
    f2_unpack(f2_fma(f2_pack(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), sl, nm), t0, t1);
    const float p0 = fast_exp2(t0), p1 = fast_exp2(t1);
    const uint64_t pr = f2_pack(p0, p1);
    if (IN_ROW)
      sum.in_row += p0 + p1;
    else
      sum.by_col[i & 1] = f2_add(sum.by_col[i & 1], pr);
    pk[i] = f2_to_bf16x2(pr);
  }
  tmem_st16(tP, pk);
}

// CUT: the window's last half tile has more than four but not all of its 64 columns (up to four come out the same in either
// order of adding up). A kernel of its own: the code by its mere presence costs full tiles 8 % (72 x 900, 24 x 64: 0.635 ->
// 0.701 ms; as a rolled loop over the cut columns or as a call it costs more).
template <int DCH, bool CUT>
__global__ void __launch_bounds__(AttnPair<DCH>::THREADS, 1)
attn_fwd_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                     const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_o,
                     const AttnFwdParams p, const int n_items_total) {
  using R = AttnPair<DCH>;
  constexpr int HD = 64 * DCH, NS = R::NS, NBQ = R::NBQ;
  constexpr bool P_OVER_S = R::COL_P == 0;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* sQ = smem;                               // [2 chains][NBQ]
  uint8_t* sK = sQ + 2 * NBQ * R::Q_BYTES;          // [NS]
  uint8_t* sV = sK + NS * R::T_BYTES;               // [NS]
  uint8_t* sO = sV + NS * R::T_BYTES;               // [2 chains]
  uint64_t* bars = reinterpret_cast<uint64_t*>(sO + 2 * R::OUT_BYTES);
  uint64_t* q_full = bars;              // [2][2]
  uint64_t* q_empty = bars + 4;         // [2][2]
  uint64_t* k_full = bars + 8;          // [NS <= 4]
  uint64_t* k_empty = bars + 12;        // [NS] both chains have taken their scores' product
  uint64_t* v_full = bars + 16;
  uint64_t* v_empty = bars + 20;
  uint64_t* s_full = bars + 24;         // [2] the chain's scores are in tensor memory
  uint64_t* s_free = bars + 26;         // [2] they have been read into registers
  uint64_t* p_full = bars + 28;         // [2] the chain's probabilities are in tensor memory (P_OVER_S: their first half)
  uint64_t* p_full2 = bars + 30;        // [2] P_OVER_S: the second half
  uint64_t* pv_done = bars + 32;        // [2] P V has completed: P may be overwritten, the accumulator is up to date
  uint64_t* turn = bars + 34;           // [2] P_OVER_S: whose products are next
  uint64_t* half = bars + 36;           // [2][4] a warp is half way through its exponentials
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 44);
  int* s_abort = reinterpret_cast<int*>(tmem_slot + 1);
  int* s_failed = s_abort + 1;      // [8] see note_failure

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int N = p.N;
  const int nfull = N / KVP, rem = N - nfull * KVP;
  const int nkv = nfull + (rem ? 1 : 0);
  const int n_last = rem ? ((rem + 15) & ~15) : KVP;      // columns computed in the last tile
  const int q_tiles = (N + TILE - 1) / TILE, n_pairs = (q_tiles + 1) >> 1;
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
    for (int i = 0; i < 4; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
    for (int i = 0; i < NS; ++i) {
      mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 2);
      mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 2);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&s_full[i], 1); mbar_init(&s_free[i], 4); mbar_init(&p_full[i], 4); mbar_init(&p_full2[i], 4);
      mbar_init(&pv_done[i], 1); mbar_init(&turn[i], 1);
    }
    for (int i = 0; i < 8; ++i) mbar_init(&half[i], 1);
    fence_barrier_init();
  }
  if (warp == 8) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_point();

  if (warp == 8) {
    // ------------------------------------------------------------ TMA producer
    if (elect_one_sync()) {
      int vi[2] = {0, 0};               // query tiles requested so far, per chain
      auto load_q = [&](const PairItem& w, int c) -> bool {
        const int qt = 2 * w.pair + c;
        if (qt >= q_tiles) return true;
        const int b = vi[c] % NBQ;
        if (!mbar_wait(&q_empty[2 * c + b], ((vi[c] / NBQ) & 1) ^ 1, p.status, ERR_TIMEOUT_ATTN)) return false;
        uint64_t* bar = &q_full[2 * c + b];
        mbar_expect_tx(bar, R::Q_BYTES);
#pragma unroll
        for (int i = 0; i < DCH; ++i)
          tma_load_4d(sQ + (c * NBQ + b) * R::Q_BYTES + i * 16384, &tm_q, bar, i * 64, w.head, qt * TILE, w.win);
        ++vi[c];
        return true;
      };
      auto load_t = [&](uint8_t* ring, uint64_t* full, uint64_t* empty, const CUtensorMap* tm, int g, const PairItem& w,
                        int j) -> bool {
        const int st = g % NS;
        if (!mbar_wait(&empty[st], ((g / NS) & 1) ^ 1, p.status, ERR_TIMEOUT_ATTN)) return false;
        mbar_expect_tx(&full[st], R::T_BYTES);
#pragma unroll
        for (int i = 0; i < DCH; ++i)
          tma_load_4d(ring + st * R::T_BYTES + i * 16384, tm, &full[st], i * 64, w.head, j * KVP, w.win);
        return true;
      };
      // K_g, then V_(g-1): the order in which their slots come free. A chain's query tile of the next item is requested
      // with that item's first K tile; where it has one buffer that waits for the last scores of the item before, so the
      // second chain, which runs half a tile later, has its request behind V.
      PairItem cur = pair_item(0, n_pairs, p.H), prev = cur;
      int it = 0, j = 0, pj = 0;
      for (int g = 0; g <= total; ++g) {
        if (g < total) {
          if (j == 0 && (!load_q(cur, 0) || (NBQ == 2 && !load_q(cur, 1)))) break;
          if (!load_t(sK, k_full, k_empty, &tm_k, g, cur, j)) break;
        }
        if (g >= 1 && !load_t(sV, v_full, v_empty, &tm_v, g - 1, prev, pj)) break;
        if (g < total) {
          if (j == 0 && NBQ == 1 && !load_q(cur, 1)) break;
          prev = cur;
          pj = j;
          if (++j == nkv) {
            j = 0;
            if (++it < n_items) cur = pair_item(it, n_pairs, p.H);
          }
        }
      }
    }
  } else if (warp == 9 || warp == 10) {
    // ------------------------------------------------------------ MMA issuer of one chain
    if (elect_one_sync()) {
      const int c = warp - 9;
      const uint32_t tS = tmem_base + c * 256, tP = tS + R::COL_P, tO = tS + R::COL_O;
      const uint32_t aQ = smem_u32(sQ) + c * NBQ * R::Q_BYTES, aK = smem_u32(sK), aV = smem_u32(sV);
      constexpr uint32_t idesc_pv = make_idesc_bf16(TILE, HD, 0, 1);
      auto has_rows = [&](int it) { return 2 * pair_item(it, n_pairs, p.H).pair + c < q_tiles; };
      int s_it = 0, s_j = 0, s_g = 0, s_t = 0, s_vi = 0;      // next scores: item, tile, number (all / own), own item
      bool s_ok = has_rows(0);
      // S = Q K_j^T. A chain without rows in an item only gives the tiles back.
      auto issue_qk = [&]() -> bool {
        const int st = s_g % NS;
        const bool last = s_j == nkv - 1;
        if (s_ok) {
          const int b = s_vi % NBQ;
          if (s_j == 0 && !mbar_wait(&q_full[2 * c + b], (s_vi / NBQ) & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
          if (!P_OVER_S && s_t > 0 && !mbar_wait(&s_free[c], (s_t - 1) & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
          if (!mbar_wait(&k_full[st], (s_g / NS) & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
          tc_fence_after();
          const uint32_t idesc = make_idesc_bf16(TILE, last ? n_last : KVP, 0, 0);
          const uint64_t dq = make_smem_desc(aQ + b * R::Q_BYTES, 0, 1024);
          const uint64_t dk = make_smem_desc(aK + st * R::T_BYTES, 0, 1024);
#pragma unroll
          for (int kk = 0; kk < 4 * DCH; ++kk) {
            const uint32_t off = ((kk >> 2) * 16384 + (kk & 3) * 32) / 16;
            umma_ss(tS, dq + off, dk + off, idesc, kk > 0);
          }
          tc_commit(&s_full[c]);
          tc_commit(&k_empty[st]);
          if (last) { tc_commit(&q_empty[2 * c + b]); ++s_vi; }
          ++s_t;
        } else {
          if (!mbar_wait(&k_full[st], (s_g / NS) & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
          mbar_arrive(&k_empty[st]);
        }
        ++s_g;
        if (++s_j == nkv) {
          s_j = 0;
          if (++s_it < n_items) s_ok = has_rows(s_it);
        }
        return true;
      };
      // With P over the scores a chain's next scores wait for its P V: the chains have to take turns, one in its products
      // while the other is in its softmax. Left alone they run in step, where their products, interleaved, finish together
      // and both softmaxes compete for the exp unit (cycles per pair of tiles at head_dim 128: 4,800; in turns 3,500).
      auto take_turn = [&](int n) { return mbar_wait(&turn[c], n & 1, p.status, ERR_TIMEOUT_ATTN); };
      bool ok = true;
      if (P_OVER_S && c == 1) ok = take_turn(0);
      ok = ok && issue_qk();
      if (P_OVER_S) mbar_arrive(&turn[1 - c]);
      int a_it = 0, a_j = 0, a_t = 0;
      bool a_ok = has_rows(0);
      for (int g = 0; g < total && ok; ++g) {
        // with columns of its own for P the next tile's scores run under this tile's softmax
        if (!P_OVER_S && s_g < total && !issue_qk()) break;
        const int st = g % NS;
        if (!mbar_wait(&v_full[st], (g / NS) & 1, p.status, ERR_TIMEOUT_ATTN)) break;
        if (a_ok) {
          if (!mbar_wait(&p_full[c], a_t & 1, p.status, ERR_TIMEOUT_ATTN)) break;
          tc_fence_after();
          // O += P_j V_j  (A = P in tensor memory, 16 columns of bf16 = 8 words per K step; B = V MN-major)
          const uint64_t dv = make_smem_desc(aV + st * R::T_BYTES, 16384, 1024);
          const int ksteps = (a_j == nkv - 1 ? n_last : KVP) / 16;
          const uint32_t acc0 = a_j > 0 ? 1u : 0u;
          if (ksteps == KVP / 16) {
#pragma unroll
            for (int kk = 0; kk < KVP / 32; ++kk) umma_ts(tO, tP + kk * 8, dv + kk * 128, idesc_pv, kk ? 1u : acc0);
            if (P_OVER_S) {
              if (!mbar_wait(&p_full2[c], a_t & 1, p.status, ERR_TIMEOUT_ATTN) || !take_turn(g + c)) break;
              tc_fence_after();
            }
#pragma unroll
            for (int kk = KVP / 32; kk < KVP / 16; ++kk) umma_ts(tO, tP + kk * 8, dv + kk * 128, idesc_pv, 1u);
          } else {
            if (P_OVER_S) {
              if (!mbar_wait(&p_full2[c], a_t & 1, p.status, ERR_TIMEOUT_ATTN) || !take_turn(g + c)) break;
              tc_fence_after();
            }
            for (int kk = 0; kk < ksteps; ++kk) umma_ts(tO, tP + kk * 8, dv + kk * 128, idesc_pv, kk ? 1u : acc0);
          }
          tc_commit(&pv_done[c]);
          tc_commit(&v_empty[st]);
          ++a_t;
        } else {
          if (P_OVER_S && !take_turn(g + c)) break;
          mbar_arrive(&v_empty[st]);
        }
        if (++a_j == nkv) {
          a_j = 0;
          if (++a_it < n_items) a_ok = has_rows(a_it);
        }
        // the scores overwrite P, which the tensor core has consumed by then: it executes in issue order
        if (P_OVER_S && s_g < total && !issue_qk()) break;
        if (P_OVER_S) mbar_arrive(&turn[1 - c]);
      }
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------ softmax: one thread = one query row of its chain
    const int c = warp >> 2, q = warp & 3;
    const int row = q * 32 + lane;
    note_failure(p.status, &s_failed[warp]);
    const uint32_t lane_addr = static_cast<uint32_t>(q * 32) << 16;
    const uint32_t tS = tmem_base + c * 256 + lane_addr, tP = tS + R::COL_P, tO = tS + R::COL_O;
    const float sl2 = p.scale_log2;
    const uint64_t sl = f2_pack(sl2, sl2);
    int t = 0;                          // tiles of this chain so far
    bool ok = true;
    float m_ref = 0.f, l = 0.f;
    auto wait_pv = [&]() -> bool {      // P V of the tile before has completed
      if (!mbar_wait(&pv_done[c], (t - 1) & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
      tc_fence_after();
      return true;
    };
    // Output rows and row statistics of an item, whose last P V has completed. A warp's rows leave as tiles of 32 through
    // shared memory (one thread a row, 16 bytes a store, would touch 32 rows with every instruction). Every lane-0 block is
    // followed by a warp barrier: the next step reads tensor memory, which takes the whole warp.
    uint8_t* stage = sO + c * R::OUT_BYTES + q * 4096;
    auto epilogue = [&](const PairItem& w) {
      const int grow = (2 * w.pair + c) * TILE + row;
      const float inv = 1.f / l;
      __nv_bfloat16* pdst = nullptr;
      if (p.push_n_local > 0 && grow < N) {
        const int owner = grow / p.push_n_local;
        pdst = reinterpret_cast<__nv_bfloat16*>(p.o_peers[owner]) +
               (static_cast<size_t>(w.win) * p.push_n_local + (grow - owner * p.push_n_local)) * p.push_ld +
               p.push_col0 + w.head * p.d;
      }
#pragma unroll 1
      for (int col = 0; col < HD && col < p.d; col += 64) {
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t v[32];
          tmem_ld32(tO + col + 32 * h, v);
          tmem_wait_ld();
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            uint32_t o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
              o[i] = pack_bf16x2(__uint_as_float(v[8 * g + 2 * i]) * inv, __uint_as_float(v[8 * g + 2 * i + 1]) * inv);
            const uint4 u = make_uint4(o[0], o[1], o[2], o[3]);
            *reinterpret_cast<uint4*>(stage + swz128(lane, 4 * h + g)) = u;
            if (pdst && col + 32 * h + 8 * g < p.d) *reinterpret_cast<uint4*>(pdst + col + 32 * h + 8 * g) = u;
          }
        }
        fence_proxy_async_smem();
        __syncwarp();
        // columns past the head's width and rows past the window's end are clipped
        if (lane == 0 && p.O) tma_store_4d(&tm_o, stage, col, w.head, (2 * w.pair + c) * TILE + q * 32, w.win);
        __syncwarp();
      }
      if (p.lse && grow < N)
        p.lse[(static_cast<size_t>(w.win) * p.H + w.head) * N + grow] = m_ref + log2f(l);
    };
    auto arrive = [&](uint64_t* bar) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };
    auto wait_s = [&]() -> bool {
      if (!mbar_wait(&s_full[c], t & 1, p.status, ERR_TIMEOUT_ATTN)) return false;
      tc_fence_after();
      return true;
    };
    // The two chains' warps of a scheduler share its exp unit. Each starts its exponentials when the other is half way
    // through its own: in step, both would wait for the unit together and leave it idle together, and nothing in the
    // hand-shakes pulls them apart (head_dim 64, without / with: 200 x 225 tokens 0.178 / 0.170 ms, 72 x 900 0.623 / 0.618).
    int turn_no = 0;
    auto their_half = [&]() -> bool {
      return (c == 0 && turn_no == 0) ||
             mbar_wait(&half[(1 - c) * 4 + q], (turn_no - (1 - c)) & 1, p.status, ERR_TIMEOUT_ATTN);
    };
    auto my_half = [&]() {
      __syncwarp();
      if (lane == 0) mbar_arrive(&half[c * 4 + q]);
      ++turn_no;
    };
    // One tile of a warp without rows: the hand-shakes only.
    auto idle_tile = [&](int j) -> bool {
      if (!wait_s()) return false;
      if (!P_OVER_S) arrive(&s_free[c]);
      if (j > 0 && !wait_pv()) return false;
      arrive(&p_full[c]);
      if (P_OVER_S) arrive(&p_full2[c]);
      if (!P_OVER_S) {
        if (!their_half()) return false;
        my_half();
      }
      ++t;
      return true;
    };
    // One tile: scores -> probabilities. `cols`: columns that the products computed (and P V reads), `fill`: first of them
    // that is past the window's end. One copy of the code serves full and partial tiles: a second, unrolled one that runs
    // once per item is not in the instruction cache when it is needed (the last tile of 900 tokens with the epilogue: 8,900
    // cycles, 4,900 with one copy).
    auto tile = [&](int j, int cols, int fill) -> bool {
      if (!wait_s()) return false;
      if (fill < KVP) {
#pragma unroll 1
        for (int k = fill & ~7; k < (cols > 64 ? KVP : cols > 32 ? 64 : 32); k += 8) {
          uint32_t x[8];
          if (k < fill) {
            tmem_ld8(tS + k, x);
            tmem_wait_ld();
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (k + i >= fill) x[i] = 0xff800000u;      // -inf: probability 0
          tmem_st8(tS + k, x);
        }
        tmem_wait_st();
      }
      uint32_t v[4][32];
#pragma unroll
      for (int h = 0; h < 4; ++h) tmem_ld32(tS + 32 * h, v[h]);      // what lies past `cols` is not looked at
      tmem_wait_ld();
      if (!P_OVER_S) arrive(&s_free[c]);
      // The reference maximum is raised as attn_fwd_kernel raises it, which sees 64 columns at a time: by the first half
      // alone, unless the second exceeds that by 2^8 (then both halves take the second's). One vote serves a tile that does
      // not raise it, the usual one.
      auto row_max = [&](const uint32_t (&x)[32], const uint32_t (&y)[32], bool both) {
        float mx[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) mx[k] = fmaxf(__uint_as_float(x[k]), __uint_as_float(x[k + 4]));
#pragma unroll
        for (int i = 8; i < 32; i += 8) {
#pragma unroll
          for (int k = 0; k < 4; ++k) mx[k] = max3(mx[k], __uint_as_float(x[i + k]), __uint_as_float(x[i + k + 4]));
        }
        if (both) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
#pragma unroll
            for (int k = 0; k < 4; ++k) mx[k] = max3(mx[k], __uint_as_float(y[i + k]), __uint_as_float(y[i + k + 4]));
          }
        }
        return fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]) * sl2;
      };
      const float max_1 = row_max(v[0], v[1], cols > 32);
      float max_2 = -INFINITY;
      if (cols > 64) max_2 = row_max(v[2], v[3], true);
      bool waited = P_OVER_S || j == 0;     // P_OVER_S: these scores were issued behind the P V of the tile before
      if (__any_sync(0xffffffffu, max3(m_ref, max_1, max_2) - m_ref > RESCALE_LOG2)) {
        float m_new = fmaxf(m_ref, max_1);
        if (!__any_sync(0xffffffffu, m_new - m_ref > RESCALE_LOG2)) m_new = m_ref;
        if (__any_sync(0xffffffffu, max_2 - m_new > RESCALE_LOG2)) m_new = fmaxf(m_new, max_2);
        if (j > 0) {
          if (!waited && !wait_pv()) return false;
          waited = true;
          const float alpha = fast_exp2(m_ref - m_new);
          rescale_tmem_rows(tO, HD, alpha);
          l *= alpha;
        }
        m_ref = m_new;
      }
      const uint64_t nm = f2_pack(-m_ref, -m_ref);
      if (!waited && !wait_pv()) return false;
      if (!P_OVER_S && !their_half()) return false;
      const bool cut_1 = CUT && fill < 64, cut_2 = CUT && fill < KVP;
      HalfSum sum_1, sum_2;
      auto half = [&](const uint32_t (&x)[32], const uint32_t (&y)[32], bool both, bool cut, HalfSum& sum, uint32_t to) {
        if (cut) {
          softmax_chunk<true>(x, sl, nm, sum, to);
          if (both) softmax_chunk<true>(y, sl, nm, sum, to + 16);
        } else {
          softmax_chunk<false>(x, sl, nm, sum, to);
          if (both) softmax_chunk<false>(y, sl, nm, sum, to + 16);
        }
      };
      half(v[0], v[1], cols > 32, cut_1, sum_1, tP);
      if (!P_OVER_S) my_half();
      if constexpr (P_OVER_S) {
        tmem_wait_st();
        arrive(&p_full[c]);
      }
      if (cols > 64) half(v[2], v[3], true, cut_2, sum_2, tP + 32);
      l += sum_1.total(cut_1);
      l += sum_2.total(cut_2);
      tmem_wait_st();
      arrive(P_OVER_S ? &p_full2[c] : &p_full[c]);
      ++t;
      return true;
    };
    for (int it = 0; it < n_items && ok; ++it) {
      const PairItem w = pair_item(it, n_pairs, p.H);
      const int qt = 2 * w.pair + c;
      if (qt >= q_tiles) {
        if (!P_OVER_S)
          for (int j = 0; j < nkv && ok; ++j) {
            ok = their_half();
            my_half();
          }
        continue;
      }
      const bool rows = qt * TILE + q * 32 < N;
      m_ref = -INFINITY;
      l = 0.f;
      if (rows) {
        for (int j = 0; j < nkv && ok; ++j) ok = tile(j, j < nfull ? KVP : n_last, j < nfull ? KVP : rem);
      } else {
        for (int j = 0; j < nkv && ok; ++j) ok = idle_tile(j);
      }
      if (!ok || !wait_pv()) break;
      if (rows && !noted(&s_failed[warp])) epilogue(w);
    }
    // the copies have been performed before their shared memory goes
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 8) tmem_dealloc(tmem_base, 512);
}

template <int DCH, bool CUT>
static int launch_attn_fwd_pair(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                                const CUtensorMap& to, const AttnFwdParams& p, cudaStream_t stream) {
  using R = AttnPair<DCH>;
  auto kern = attn_fwd_pair_kernel<DCH, CUT>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, R::SMEM) != cudaSuccess) return -20;
    configured = true;
  }
  const int pairs = ((p.N + TILE - 1) / TILE + 1) / 2;
  const long long items = static_cast<long long>(pairs) * p.H * p.n_win;
  const int nkv = (p.N + KVP - 1) / KVP;
  if (items > 0x3fffffff || items * nkv > 0x3fffffffll * num_sms()) return -23;
  const int n = static_cast<int>(items), grid = n < num_sms() ? n : num_sms();
  return launch_chained(kern, grid, R::THREADS, R::SMEM, stream, tq, tk, tv, to, p, n);
}

}  // namespace aeris
