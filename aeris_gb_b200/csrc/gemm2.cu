// Two-CTA variant of the persistent tcgen05 GEMM: a thread-block cluster of two CTAs (one SM pair) computes one
// 256 x 256 output tile with `tcgen05.mma.cta_group::2`. Each CTA stages its own 128 rows of A and only HALF of the
// B tile (128 of the 256 columns), so the shared-memory operand traffic per FLOP is a third lower than in the
// one-CTA 128 x 256 kernel, which is bound by exactly that traffic (73 % tensor-pipe utilisation).
//
// Every CTA issues its own plain TMA loads (no load is shared between the two CTAs). Cross-CTA signalling:
//   * stage filled : both CTAs' TMA loads credit their bytes to ONE barrier in the leader CTA (loads issued with
//                    cta_group::2, barrier addressed through the cluster window), on which the MMA thread waits;
//   * stage free   : one `tcgen05.commit` arrives on the same barrier in both CTAs (commit with a CTA mask);
//   * accumulator ready: same two-CTA commit; accumulator drained: both CTAs' epilogue warps arrive on the leader.
// Every wait is bounded and every role falls through to one final cluster barrier, so a time-out in one CTA can not
// leave its peer waiting forever. Nothing is under way any more when a CTA gets there: each role waits for what it started
// and nobody took (operand tiles, requests ahead, products), whatever it was that ended its loop.
#include "common.cuh"
#include "api.h"
#include "host.h"
#include "gemm_epilogue.cuh"
#include "gemm_ag.cuh"

#include <stdio.h>
#include <stdlib.h>

namespace aeris {

constexpr int G2_BM = 128;       // rows per CTA (256 per pair)
constexpr int G2_BN = 256;
constexpr int G2_BK = 64;
constexpr int G2_STAGES = 6;
constexpr int G2_A_BYTES = G2_BM * G2_BK * 2;         // 16 KB
constexpr int G2_B_BYTES = (G2_BN / 2) * G2_BK * 2;   // 16 KB: this CTA's half of B
constexpr int G2_STAGE_BYTES = G2_A_BYTES + G2_B_BYTES;
// Epilogue warps and ring depth. With a short reduction the epilogue of a tile takes longer than its products, so the
// heavier local epilogues then run on eight warps, two per 32 rows with half of the columns each, for the price of one ring
// stage (their staging buffers; see aeris_gemm_bf16_2cta for the line). Everything else keeps four warps and six stages.
template <int EW> struct G2Layout {
  static constexpr int STAGES = EW == 8 ? G2_STAGES - 1 : G2_STAGES;
  static constexpr int PUSH_OFF = STAGES * G2_STAGE_BYTES + 1024;     // staging of the epilogues, 8 KB per warp
  static constexpr int SMEM = PUSH_OFF + EW * PUSH_STAGE_BYTES + 1024;
  static constexpr int THREADS = 64 + EW * 32;
};
static_assert(G2Layout<4>::SMEM <= 227 * 1024 && G2Layout<8>::SMEM <= 227 * 1024, "shared memory");

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t smem_addr, uint32_t cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(cta));
  return r;
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-D tiled TMA load for a CTA pair: the data lands in THIS CTA's shared memory, the byte count is credited to the
// barrier at `bar_cluster_addr`, which may live in the other CTA of the pair (the leader's "stage full" barrier).
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* m, uint32_t bar_cluster_addr,
                                                 int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
      "[%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar_cluster_addr), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc2(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish2() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc2(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Arrive on the barrier at the same shared-memory offset in every CTA named by `mask` once all prior tcgen05 ops of
// this thread have completed.
__device__ __forceinline__ void tc_commit2_mc(uint64_t* bar, uint16_t mask) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(mask)
      : "memory");
}
__device__ __forceinline__ void umma2_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t"
      ".reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
      "}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// AG = true: the A operand is all-gathered over peer memory inside the kernel (GemmParams::ag_*): m-tiles are visited
// starting with this rank's own row chunk while two extra warps (6, 7) of every CTA push that chunk into the peers'
// buffers; the producer of each CTA waits for the chunks its 128 rows come from. The grid is then always the full
// number of CTA pairs, so that every call adds the same amount to the arrival counters.
template <int A_MN, int B_MN, int EW, bool AG = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(G2Layout<EW>::THREADS + (AG ? AG_COPY_THREADS : 0), 1)
gemm2_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
             const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ CUtensorMap tmap_x, const GemmParams p) {
  static_assert(!AG || EW == 4, "the copier warps follow four epilogue warps");
  using LY = G2Layout<EW>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + LY::STAGES * G2_STAGE_BYTES);
  uint64_t* empty_bar = full_bar + LY::STAGES;
  uint64_t* tfull_bar = empty_bar + LY::STAGES;       // [2]
  uint64_t* tempty_bar = tfull_bar + 2;              // [2], leader only: one arrival per epilogue warp of both CTAs
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);

  // AG: the last operand stage is the copier's ring (two 16 KB bulk-copy buffers), with its barriers behind tmem_slot
  // (the reduce-scatter epilogue gives up the same stage: its fourth warp stages its rows there)
  // and so does the gated residual on eight warps where it requests its second operand ahead, which it gains from while its
  // tile's products are short (us without / with, in turn: 28800 x 512 x 512 36.8 / 31.0, x 768 x 768 57.0 / 48.3, x
  // 1024 x 1024 86.0 / 73.2, 64800 x 512 x 512 71.5 / 61.1; a few per cent at 28800 x 768 x 1536 79.8 / 76.2 and 64800 x
  // 1536 x 1536 321 / 308; 28800 x 768 x 2048 94.3 / 97.7: the ring's fifth stage is worth more).
  const bool ahead = EW == 8 && p.staged_out;
  const bool u_ahead = ahead && p.epi == EPI_SWIGLU_BWD, r_ahead = ahead && p.epi == EPI_GATE_RESID && !p.aux && p.K <= 1024;
  const int STAGES = (r_ahead || (EW == 4 && (AG || p.epi == EPI_RS_PUSH))) ? LY::STAGES - 1 : LY::STAGES;
  [[maybe_unused]] uint8_t* ag_ring = smem + (LY::STAGES - 1) * G2_STAGE_BYTES;
  [[maybe_unused]] uint64_t* ag_bars = reinterpret_cast<uint64_t*>(smem + LY::STAGES * G2_STAGE_BYTES + 256);
  uint64_t* u_bars = reinterpret_cast<uint64_t*>(smem + LY::STAGES * G2_STAGE_BYTES + 320);     // [EW][2]

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t crank = cluster_ctarank();          // 0 = leader (issues the MMAs)
  const int cluster_id = blockIdx.x >> 1;
  const int n_clusters = gridDim.x >> 1;

  const int m_tiles = (p.M + 2 * G2_BM - 1) / (2 * G2_BM);
  const int n_tiles = (p.N + G2_BN - 1) / G2_BN;     // the last tile may be half empty (N a multiple of 128)
  const int kb_total = (p.K + G2_BK - 1) / G2_BK;
  const int kb_per_split = (kb_total + p.k_splits - 1) / p.k_splits;
  const int total_tiles = m_tiles * n_tiles * p.k_splits;
  const int tm_rot = AG ? (p.ag_rank * p.ag_rows) / (2 * G2_BM) : p.tm_rot;
  // Order of the tiles of one K split. The CTA pairs at work together cover `group_m` m-tiles by about 74 / group_m
  // n-tiles instead of one or two m-tiles by all n-tiles: with a wide B (w1 of dim 5120 is 280 MB, more than L2) the
  // pairs would otherwise stream all of B from HBM once per wave. group_m = 1 keeps n fastest, which the peer-memory
  // variants rely on (rows in order of arrival). 28800 x 27392 x 5120 with the SwiGLU
  // epilogue: 7.60 -> 6.34 ms; its data gradient 7.28 -> 5.40 ms; no change where B fits L2.
  auto tile_mn = [&](int mn, int& tm, int& tn) {
    if (p.group_m <= 1) {
      tm = mn / n_tiles;
      tn = mn - tm * n_tiles;
      tm = (tm + tm_rot) % m_tiles;
    } else {
      const int g = mn / (p.group_m * n_tiles), in = mn - g * p.group_m * n_tiles;
      const int gm = min(p.group_m, m_tiles - g * p.group_m);
      tn = in / gm;
      tm = g * p.group_m + in - tn * gm;
    }
  };

  if (threadIdx.x == 0) {
    prefetch_tmap(&tmap_a);
    prefetch_tmap(&tmap_b);
    for (int s = 0; s < LY::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2 * EW; ++i) mbar_init(&u_bars[i], 1);
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 2 * EW);
      if constexpr (AG) mbar_init(&ag_bars[a], 1);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc2(tmem_slot, 2 * G2_BN);
    tmem_relinquish2();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();       // both CTAs' barriers are initialised and TMEM is allocated before anyone signals
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  chain_point();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (each CTA loads its own operands)
    if (elect_one_sync()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      [[maybe_unused]] uint32_t ag_ready = 0;
      for (int tile = cluster_id; tile < total_tiles && ok; tile += n_clusters) {
        const int split = tile / (m_tiles * n_tiles);
        const int mn = tile - split * (m_tiles * n_tiles);
        int tm, tn;
        tile_mn(mn, tm, tn);
        const int kb0 = split * kb_per_split;
        const int kb1 = min(kb_total, kb0 + kb_per_split);
        const int m0 = tm * 2 * G2_BM + crank * G2_BM;
        if constexpr (AG) {
          if (m0 < p.M && !ag_wait_rows(p, m0, m0 + G2_BM, ag_ready)) { ok = false; break; }
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait_poll(&empty_bar[stage], phase ^ 1, p.status, ERR_TIMEOUT_EMPTY)) { ok = false; break; }
          uint8_t* sa = smem + stage * G2_STAGE_BYTES;
          uint8_t* sb = sa + G2_A_BYTES;
          // one "stage full" barrier per pair, in the leader: it expects the bytes of both CTAs' copies
          if (crank == 0) mbar_expect_tx(&full_bar[stage], 2 * G2_STAGE_BYTES);
          const uint32_t fb = map_to_cta(smem_u32(&full_bar[stage]), 0);
          if (A_MN == 0) {
            tma_load_2d_pair(sa, &tmap_a, fb, kb * G2_BK, m0);
          } else {
#pragma unroll
            for (int j = 0; j < G2_BM / 64; ++j)
              tma_load_2d_pair(sa + j * 8192, &tmap_a, fb, m0 + j * 64, kb * G2_BK);
          }
          if (B_MN == 0) {
            // rows of B for this CTA's half: plain tiles take 128 consecutive rows; the SwiGLU layouts pair the
            // leader with the gate rows and the peer with the up rows of the same features
            const int r0 = tn * p.b_tile_stride + (crank ? p.b_half_off : 0);
            tma_load_2d_pair(sb, &tmap_b, fb, kb * G2_BK, r0);
          } else {
#pragma unroll
            for (int j = 0; j < 2; ++j)
              tma_load_2d_pair(sb + j * 8192, &tmap_b, fb, tn * G2_BN + (crank * 2 + j) * 64, kb * G2_BK);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
      // the tiles that the issuer did not take, of both CTAs: their bytes are on the leader's barriers (a stage never filled
      // counts as there)
      for (int s = 0; s < STAGES && !ok && crank == 0; ++s) {
        if (--stage < 0) { stage = STAGES - 1; phase ^= 1; }
        if (!mbar_wait_poll(&full_bar[stage], phase, nullptr, 0)) break;
      }
    }
  } else if (warp == 1) {
    if (elect_one_sync()) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      if (crank == 0) {
        // -------------------------------------------------------- leader: MMA issuer for the CTA pair
        constexpr uint32_t idesc = make_idesc_bf16(2 * G2_BM, G2_BN, A_MN, B_MN);
        int acc = 0;
        uint32_t acc_phase = 0;
        for (int tile = cluster_id; tile < total_tiles && ok; tile += n_clusters) {
          const int split = tile / (m_tiles * n_tiles);
          const int kb0 = split * kb_per_split;
          const int kb1 = min(kb_total, kb0 + kb_per_split);
          if (!mbar_wait_poll(&tempty_bar[acc], acc_phase ^ 1, p.status, ERR_TIMEOUT_TMEM_EMPTY)) { ok = false; break; }
          tc_fence_after();
          const uint32_t tmem_acc = tmem_base + acc * G2_BN;
          for (int kb = kb0; kb < kb1; ++kb) {
            if (!mbar_wait_poll(&full_bar[stage], phase, p.status, ERR_TIMEOUT_FULL)) { ok = false; break; }
            tc_fence_after();
            const uint32_t sa = smem_u32(smem + stage * G2_STAGE_BYTES);
            const uint32_t sb = sa + G2_A_BYTES;
#pragma unroll
            for (int kk = 0; kk < G2_BK / 16; ++kk) {
              const uint64_t adesc = A_MN ? make_smem_desc(sa + kk * 2048, 8192, 1024)
                                          : make_smem_desc(sa + kk * 32, 0, 1024);
              const uint64_t bdesc = B_MN ? make_smem_desc(sb + kk * 2048, 8192, 1024)
                                          : make_smem_desc(sb + kk * 32, 0, 1024);
              umma2_ss(tmem_acc, adesc, bdesc, idesc, (kb > kb0 || kk > 0) ? 1u : 0u);
            }
            tc_commit2_mc(&empty_bar[stage], 0x3);     // frees the stage in both CTAs
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
          if (!ok) break;
          tc_commit2_mc(&tfull_bar[acc], 0x3);         // accumulator ready in both CTAs
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
        // the last products have completed: an epilogue that gave up has not waited for them
        if (--stage < 0) { stage = STAGES - 1; phase ^= 1; }
        mbar_wait_poll(&empty_bar[stage], phase, nullptr, 0);
      }
    }
  } else if (AG && warp >= 6) {
    // ------------------------------------------------------------ all-gather copier (warp 6 of both CTAs)
    if constexpr (AG) {
      if (elect_one_sync()) ag_push_chunk(p, ag_ring, ag_bars);
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2 .. 1 + EW of both CTAs)
    const int q = warp & 3, part = (warp - 2) >> 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    const uint32_t leader_tempty0 = map_to_cta(smem_u32(&tempty_bar[0]), 0);
    [[maybe_unused]] uint8_t* ubuf = smem + (LY::STAGES - 1) * G2_STAGE_BYTES + (warp - 2) * SWIGLU_U_BYTES;
    // two buffers per warp in turn: gate and up columns of a step come in, their gradients leave from the same place
    [[maybe_unused]] uint64_t* u_bar = &u_bars[2 * (warp - 2)];
    [[maybe_unused]] uint8_t* ustage = smem + LY::PUSH_OFF + (part * 4 + q) * PUSH_STAGE_BYTES;
    [[maybe_unused]] int u_n = 0, u_m = 0;         // steps requested, taken
    [[maybe_unused]] auto u_request = [&](int row0, int col) {
      if (lane == 0) {
        uint8_t* dst = ustage + (u_n & 1) * SWIGLU_U_BYTES;
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");      // the gradients before have left it
        mbar_expect_tx(u_bar + (u_n & 1), SWIGLU_U_BYTES);
        tma_load_2d(dst, &tmap_x, u_bar + (u_n & 1), col, row0);
        tma_load_2d(dst + SWIGLU_U_BYTES / 2, &tmap_x, u_bar + (u_n & 1), p.swiglu_f + col, row0);
      }
      ++u_n;
      __syncwarp();
    };
    // first step of the next tile from `tile` on that has columns for this warp (the last tile of a row may be half empty)
    [[maybe_unused]] auto request_tile = [&](int tile) {
      for (; tile < total_tiles; tile += n_clusters) {
        int tm, tn;
        tile_mn(tile, tm, tn);
        const int c = part * (G2_BN / 2);
        if (tn * G2_BN + c >= p.N) continue;
        if (u_ahead)
          u_request(tm * 2 * G2_BM + crank * G2_BM + q * 32, tn * G2_BN + c);
        else
          resid_request(ubuf, p, tm * 2 * G2_BM + crank * G2_BM + q * 32, tn * G2_BN + c, lane);
        break;
      }
    };
    if constexpr (EW == 8) {
      if (u_ahead || r_ahead) request_tile(cluster_id);
    }
    for (int tile = cluster_id; tile < total_tiles && ok; tile += n_clusters) {
      const int split = tile / (m_tiles * n_tiles);
      const int mn = tile - split * (m_tiles * n_tiles);
      int tm, tn;
      tile_mn(mn, tm, tn);
      // the warp decides as one: what it does after giving up takes all lanes
      ok = __all_sync(0xffffffffu, mbar_wait_poll(&tfull_bar[acc], acc_phase, p.status, ERR_TIMEOUT_TMEM_FULL));
      if (!ok) break;
      tc_fence_after();
      const int row = tm * 2 * G2_BM + crank * G2_BM + q * 32 + lane;
      const uint32_t taddr = tmem_base + acc * G2_BN + (static_cast<uint32_t>(q * 32) << 16);
      const bool kempty = (split * kb_per_split) >= kb_total;
      uint8_t* stg = smem + LY::PUSH_OFF + (part * 4 + q) * PUSH_STAGE_BYTES;
      if (p.epi == EPI_RS_PUSH)     // 8704-byte linear stages: three in the push area, the fourth in the freed operand stage
        stg = (q < 3) ? smem + LY::PUSH_OFF + q * RS_STAGE_BYTES : smem + (LY::STAGES - 1) * G2_STAGE_BYTES;
      bool done = false;
      if constexpr (EW == 8) {
        if (u_ahead) {
          const int c_hi = min((part + 1) * (G2_BN / 2), p.N - tn * G2_BN);
          const int row0 = row - lane;
#pragma unroll 1
          for (int c = part * (G2_BN / 2); c < c_hi; c += 32) {
            uint4 g4[4], u4[4];
            ok = mbar_wait_warp(u_bar + (u_m & 1), (u_m >> 1) & 1, p.status, ERR_TIMEOUT_FULL);
            if (!ok) break;
            uint8_t* buf = ustage + (u_m & 1) * SWIGLU_U_BYTES;
            uint8_t* mine = buf + lane * 64;
            ++u_m;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint8_t* src = mine + ((i ^ ((lane >> 1) & 3)) << 4);
              g4[i] = *reinterpret_cast<const uint4*>(src);
              u4[i] = *reinterpret_cast<const uint4*>(src + SWIGLU_U_BYTES / 2);
            }
            if (c + 32 < c_hi)
              u_request(row0, tn * G2_BN + c + 32);
            else
              request_tile(tile + n_clusters);
            uint32_t v[32], og[16], ou[16];
            tmem_ld32(taddr + c, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t gw[4] = {g4[i].x, g4[i].y, g4[i].z, g4[i].w}, uw[4] = {u4[i].x, u4[i].y, u4[i].z, u4[i].w};
#pragma unroll
              for (int j = 0; j < 4; ++j)
                swiglu_bwd_pair(v[8 * i + 2 * j], v[8 * i + 2 * j + 1], gw[j], uw[j], og[4 * i + j], ou[4 * i + j]);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              uint8_t* dst = mine + ((i ^ ((lane >> 1) & 3)) << 4);
              *reinterpret_cast<uint4*>(dst) = make_uint4(og[4 * i], og[4 * i + 1], og[4 * i + 2], og[4 * i + 3]);
              *reinterpret_cast<uint4*>(dst + SWIGLU_U_BYTES / 2) =
                  make_uint4(ou[4 * i], ou[4 * i + 1], ou[4 * i + 2], ou[4 * i + 3]);
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) {
              if (row0 < p.M) {
                tma_store_2d(&tmap_c, buf, tn * G2_BN + c, row0);
                tma_store_2d(&tmap_c, buf + SWIGLU_U_BYTES / 2, p.swiglu_f + tn * G2_BN + c, row0);
              }
              asm volatile("cp.async.bulk.commit_group;" ::: "memory");
            }
            __syncwarp();
          }
          if (!ok) break;
          done = true;
        } else if (r_ahead) {
          const TileOut to{stg, lane};
          const float* gate = p.gate + static_cast<size_t>(min(row, p.M - 1) / p.rows_per_gate) * p.ld_gate + tn * G2_BN;
          const int c_hi = min((part + 1) * (G2_BN / 2), p.N - tn * G2_BN);
#pragma unroll 1
          for (int c = part * (G2_BN / 2); c < c_hi; c += 64) {
            uint4 x[8];
            resid_take(ubuf, lane, x);
            if (c + 64 < c_hi)
              resid_request(ubuf, p, row - lane, tn * G2_BN + c + 64, lane);
            else
              request_tile(tile + n_clusters);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t v[32], o[16];
              tmem_ld32(taddr + c + 32 * h, v);
              tmem_wait_ld();
              const float4* gsrc = reinterpret_cast<const float4*>(gate + c + 32 * h);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const uint32_t rr[4] = {x[4 * h + i].x, x[4 * h + i].y, x[4 * h + i].z, x[4 * h + i].w};
                const float4 ga = gsrc[2 * i], gb = gsrc[2 * i + 1];
                const float gg[8] = {ga.x, ga.y, ga.z, ga.w, gb.x, gb.y, gb.z, gb.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                  const float2 r2 = unpack_bf16x2(rr[j]);
                  o[4 * i + j] = pack_bf16x2(fmaf(gg[2 * j], __uint_as_float(v[8 * i + 2 * j]), r2.x),
                                             fmaf(gg[2 * j + 1], __uint_as_float(v[8 * i + 2 * j + 1]), r2.y));
                }
              }
              if (h == 0) to.wait_one();
              to.put((c >> 6) & 1, h, o);
              if (h == 1) to.send((c >> 6) & 1, &tmap_c, tn * G2_BN + c, row - lane, p.M);
            }
          }
          done = true;
        }
      }
      if (!done) gemm_epilogue_row<G2_BN>(p, taddr, row, row < p.M, tn, kempty, stg, part, EW / 4,
                                          p.staged_out ? &tmap_c : nullptr, &tmap_x);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(leader_tempty0 + acc * 8);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    // the bulk copies of the reduce-scatter push have been performed before this thread leaves (the owners read
    // their slots after a rank barrier that follows this kernel in the stream)
    if (p.epi == EPI_RS_PUSH) rs_stage_drain();
    if (p.staged_out) TileOut{nullptr, lane}.drain();
    if constexpr (EW == 8) {       // after a time-out: what was requested ahead and nobody took
      asm volatile("cp.async.wait_all;" ::: "memory");
      for (; u_m < u_n; ++u_m) mbar_wait_warp(u_bar + (u_m & 1), (u_m >> 1) & 1, p.status, ERR_TIMEOUT_FULL);
    }
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();       // nobody leaves while the pair may still touch its shared memory or TMEM
  tc_fence_after();
  if (warp == 1) tmem_dealloc2(tmem_base, 2 * G2_BN);
}

template <int A_MN, int B_MN, int EW, bool AG = false>
static int launch_gemm2(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p_in, cudaStream_t stream,
                        const CUtensorMap* tc = nullptr, const CUtensorMap* tx = nullptr) {
  static bool configured = false;
  GemmParams p = p_in;
  constexpr int THREADS = G2Layout<EW>::THREADS + (AG ? AG_COPY_THREADS : 0), SMEM = G2Layout<EW>::SMEM;
  auto kern = gemm2_kernel<A_MN, B_MN, EW, AG>;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess) return -20;
    configured = true;
  }
  const int m_tiles = (p.M + 2 * G2_BM - 1) / (2 * G2_BM);
  const int mn_tiles = m_tiles * ((p.N + G2_BN - 1) / G2_BN);
  // persistent grid = the number of CTA pairs the device can actually hold at once
  static int max_clusters = 0;
  if (max_clusters == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(num_sms(), 1, 1);
    cfg.blockDim = dim3(THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n <= 0) n = num_sms() / 2;
    max_clusters = n;
    if (getenv("AERIS_DEBUG")) fprintf(stderr, "gemm2: max active clusters %d\n", n);
  }
  int clusters = max_clusters;
  if (p.k_splits <= 0) p.k_splits = choose_k_splits(mn_tiles, (p.K + G2_BK - 1) / G2_BK, clusters, 64, -p.k_splits);
  const int tiles = mn_tiles * p.k_splits;
  if (tiles < clusters && !AG) clusters = tiles;
  if (AG) p.ag_expect *= static_cast<unsigned>(2 * clusters);   // came in as the call index
  if constexpr (AG) {          // waits for its peers: nothing of it starts before its turn
    kern<<<2 * clusters, THREADS, SMEM, stream>>>(ta, tb, tc ? *tc : ta, tx ? *tx : ta, p);
    return cudaGetLastError() == cudaSuccess ? 0 : -21;
  }
  return launch_chained(kern, 2 * clusters, THREADS, SMEM, stream, ta, tb, tc ? *tc : ta, tx ? *tx : ta, p);
}

}  // namespace aeris

using namespace aeris;

// Same contract as aeris_gemm_bf16 (api.h); N must be a multiple of 128 (of 256 for the SwiGLU forward epilogues, whose
// tiles pair gate and up columns).
static int gemm_two_cta(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc, int a_mn,
                        int b_mn, int epi, const void* resid, int ldr, const float* gate, int rows_per_gate, int ld_gate,
                        void* aux, int ld_aux, int swiglu_f, int k_splits, int* status, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0) return -1;
  const bool swiglu_fwd = (epi == EPI_SWIGLU || epi == EPI_SWIGLU_BOTH);
  if (N % (swiglu_fwd ? G2_BN : G2_BN / 2) != 0) return -2;
  if (swiglu_fwd && b_mn) return -3;
  if (k_splits < 1 && epi != EPI_ACC_F32) k_splits = 1;
  if (k_splits > 1 && epi != EPI_ACC_F32) return -4;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.epi = epi; p.C = C; p.ldc = ldc;
  p.resid = reinterpret_cast<const __nv_bfloat16*>(resid); p.ldr = ldr;
  p.gate = gate; p.rows_per_gate = rows_per_gate > 0 ? rows_per_gate : M; p.ld_gate = ld_gate;
  p.aux = reinterpret_cast<__nv_bfloat16*>(aux); p.ld_aux = ld_aux;
  p.k_splits = k_splits; p.status = status; p.swiglu_f = swiglu_f; p.group_m = 8;
  {
    static const int staged_red = [] { const char* e = getenv("AERIS_GEMM_STAGED_RED"); return e ? atoi(e) : 0; }();
    p.staged_red = staged_red;
  }
  if (swiglu_fwd) { p.b_tile_stride = G2_BN / 2; p.b_half_off = swiglu_f; }
  else            { p.b_tile_stride = G2_BN;     p.b_half_off = G2_BN / 2; }
  CUtensorMap ta, tb;
  int r;
  if (!a_mn) r = make_tmap_2d_bf16(&ta, A, K, M, lda, G2_BK, G2_BM);
  else       r = make_tmap_2d_bf16(&ta, A, M, K, lda, 64, G2_BK);
  if (r) return r;
  if (!b_mn) {
    const uint64_t brows = swiglu_fwd ? static_cast<uint64_t>(2) * swiglu_f : static_cast<uint64_t>(N);
    r = make_tmap_2d_bf16(&tb, B, K, brows, ldb, G2_BK, G2_BN / 2);
  } else {
    r = make_tmap_2d_bf16(&tb, B, N, K, ldb, 64, G2_BK);
  }
  if (r) return r - 100;
  // bf16 outputs leave as tiles of 32 rows (TileOut; on eight warps the SwiGLU backward has narrower ones, see
  // SWIGLU_U_BYTES). AERIS_GEMM_STAGED_OUT=0 selects direct stores, one 16-byte piece per row and instruction.
  const bool heavy = epi == EPI_SWIGLU_BOTH || epi == EPI_SWIGLU_BWD || epi == EPI_GATE_RESID;
  const bool ew8 = (heavy && K <= (epi == EPI_SWIGLU_BWD ? 2560 : 2048)) || (epi == EPI_STORE && K <= 1024);
  CUtensorMap tc = ta, tx = ta;
  static const int staged = [] { const char* e = getenv("AERIS_GEMM_STAGED_OUT"); return e ? atoi(e) : 1; }();
  p.staged_out = staged && !a_mn && (heavy || epi == EPI_STORE || epi == EPI_SWIGLU) && !(epi == EPI_GATE_RESID && aux);
  if (p.staged_out) {
    const uint64_t two_f = 2 * static_cast<uint64_t>(swiglu_f);
    if (epi == EPI_SWIGLU_BWD && ew8) {
      if ((r = make_tmap_2d_sw64_bf16(&tc, C, two_f, M, ldc, 32, 32))) return r - 200;
      if ((r = make_tmap_2d_sw64_bf16(&tx, resid, two_f, M, ldr, 32, 32))) return r - 300;
    } else {
      const uint64_t cols = epi == EPI_SWIGLU_BWD ? two_f : swiglu_fwd ? swiglu_f : N;
      if ((r = make_tmap_2d_bf16(&tc, C, cols, M, ldc, 64, 32))) return r - 200;
      if (epi == EPI_SWIGLU_BOTH && (r = make_tmap_2d_bf16(&tx, aux, two_f, M, ld_aux, 64, 32))) return r - 300;
    }
  }
  // Eight epilogue warps where the epilogue takes longer than the products of a tile. Four warps and six stages against
  // eight and five, us, held for 0.6 s (1.2-1.8 GHz under the power cap): gated residual 28800 x 768 x 768 62 / 53, 64800 x
  // 1536 x 1536 311 / 284, 28800 x 2048 x 2048 217 / 210, x 2304 x 2304 255 / 256, x 3072 x 3072 424 / 436; SwiGLU backward
  // 64800 x 4096 x 1536 1106 / 985, 28800 x 5376 x 2048 735 / 690, x 6144 x 2304 885 / 832, x 8192 x 3072 1334 / 1321;
  // SwiGLU with the raw columns 28800 x 4096 x 768 220 / 191, x 8192 x 1536 615 / 611, x 10752 x 2048 999 / 1035, x 12288 x
  // 2304 1270 / 1309. The raw columns lose below the line at 2048.
  // Plain store 28800 x 2304 x 768 104 / 98, x 3072 x 1024 158 / 157, x 3840 x 1280 222 / 232. Weight gradients (a_mn) lose
  // a few per cent. Since then the SwiGLU backward and the gated residual on eight warps request their second operand ahead
  // (registers for that spilled; see SWIGLU_U_BYTES), and the SwiGLU backward's line moved up. In turn, 1.2-1.5 GHz:
  // 28800 x 5376 x 2048 712 / 684, x 6144 x 2304 1017 / 810, x 6400 x 2432 1094 / 897, x 6912 x 2560 1167 / 1031; it would
  // gain further up (x 7680 x 2816 1376 / 1255), but no more at x 8192 x 3072 1469 / 1478.
  if (a_mn) return b_mn ? launch_gemm2<1, 1, 4>(ta, tb, p, stream) : launch_gemm2<1, 0, 4>(ta, tb, p, stream);
  if (b_mn)
    return ew8 ? launch_gemm2<0, 1, 8>(ta, tb, p, stream, &tc, &tx) : launch_gemm2<0, 1, 4>(ta, tb, p, stream, &tc, &tx);
  return ew8 ? launch_gemm2<0, 0, 8>(ta, tb, p, stream, &tc, &tx) : launch_gemm2<0, 0, 4>(ta, tb, p, stream, &tc, &tx);
}

extern "C" int aeris_gemm_bf16_2cta(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb,
                                    int ldc, int a_mn, int b_mn, int epi, const void* resid, int ldr,
                                    const float* gate, int rows_per_gate, void* aux, int ld_aux, int swiglu_f,
                                    int k_splits, int* status, void* stream) {
  return gemm_two_cta(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, epi, resid, ldr, gate, rows_per_gate, N, aux, ld_aux,
                      swiglu_f, k_splits, status, stream);
}

// Which kernel takes a product of N = n * 128 columns: CTA pairs on tiles of 256 x 256, whose last one may be half empty,
// or single CTAs, on tiles of 128 x 128 for stores, 256 wide where N allows it for SwiGLU and accumulating products. us,
// bursts, one CTA / pairs:
//   * plain and gated stores: a wave of pairs takes 1.2 to 1.4 times as long as one of single CTAs, so the numbers of waves
//     decide. 12150 x 384 x 1152 13.1 / 16.7 (2 and 2 waves), 4096 x 1152 x 3456 28.6 / 39.1 (2, 2), 28800 x 384 x 384
//     26.2 / 21.8 (5, 4), 12150 x 1152 x 1152 51.0 / 50.5 (6, 4), 12150 x 640 x 640 22.6 / 16.4 (4, 2), 4096 x 1664 x 4992
//     60.9 / 63.0 (3, 2), 28800 x 896 x 896 87.5 / 59.0 (11, 7); one wave of either: 3600 x 512 x 512 5.6 / 8.8.
//   * SwiGLU backward: only the pairs' kernel requests its second operand ahead. 4096 x 384 x 128 9.8 / 9.8, 12150 x 896 x
//     384 44.1 / 28.3, 64800 x 3456 x 1664 1179 / 669.
//   * SwiGLU forward that also stores the raw columns: the pairs' tiled stores. 4096 x 1024 x 256 7.9 / 8.2, 12150 x 1792 x
//     384 38.6 / 26.0, 57600 x 4096 x 768 469 / 321; only at the very smallest one CTA, 4096 x 512 x 128 5.4 / 7.3
//     (pairs take that one too: where the line would lie has not been measured).
//   * SwiGLU forward without the raw columns: its tiles halve on the way out, and short sums leave the epilogue as the
//     bound, which every CTA of its own overlaps better. 14400 x 1024 x 256 13.8 / 17.2, 64800 x 1024 x 384 59 / 67,
//     28800 x 3072 x 384 76.6 / 83.6; held for 0.25 s 64800 x 2048 x 384 120 / 126, x 2048 x 512 146 / 144.
//   * weight gradients (sums over tokens, split where tiles are few): with a half-empty last tile the pairs win by their
//     longer sums. 1152 x 384 x 12150 14.5 / 18.5, x 28800 31.8 / 32.0, x 64800 69.7 / 63.0; 384 x 384 x 28800 25.2 / 21.6;
//     1664 x 1664 x 12150 88.0 / 79.1, x 4096 39.0 / 43.9.
static bool pairs_pay(int M, int N, int K, int epi) {
  if (epi == EPI_SWIGLU) return K > 384;
  if (epi == EPI_SWIGLU_BOTH || epi == EPI_SWIGLU_BWD) return true;
  if (epi == EPI_ACC_F32) return N % G2_BN == 0 || N >= 2048 || K >= 20000 || static_cast<double>(M) * N * K >= 2e10;
  const long long one = static_cast<long long>((M + 127) / 128) * (N / 128);
  const long long two = static_cast<long long>((M + 255) / 256) * ((N + 255) / 256);
  const int sms = num_sms(), pairs = sms > 1 ? sms / 2 : 1;
  return 5 * ((two + pairs - 1) / pairs) <= 4 * ((one + sms - 1) / sms);
}
// A weight gradient that asks for slices (k_splits < 0) gets them from either kernel only as far as they are free, and a
// quarter of the tiles leaves less room for free ones: of 60 asked for at 1152 x 384 x 53550 single CTAs make 27 of 1,984
// rows, pairs 7 of 7,680; of 240 at 384 x 384 210 of 256 and 18 of 3,008. The error of a sum grows with its slice's rows, so
// between the lines above pairs take it only where their slices are no longer. (k_splits = 0: four slices on single CTAs, at
// least as many on pairs.) Error against 64 bits and us, single CTAs / pairs: the first 2.0e-6 / 8.5e-6 and 57 / 54, the
// second 3.5e-7 / 3.2e-6 and 70 / 29, 1792 x 384 x 28800 with 240 7.3e-7 / 6.3e-6 and 58 / 43, 1152 x 384 x 20250 with 16
// 1.3e-6 / 3.1e-6 and 25 / 28.
static bool slices_stay(int M, int N, int K, int k_splits, int sms) {
  if (k_splits >= 0 || N % G2_BN == 0 || N >= 2048) return true;
  const int kb = (K + G2_BK - 1) / G2_BK, pairs = sms > 1 ? sms / 2 : 1;
  const int one = choose_k_splits(((M + 127) / 128) * (N / 128), kb, sms, 4, -k_splits);
  const int two = choose_k_splits(((M + 255) / 256) * ((N + G2_BN - 1) / G2_BN), kb, pairs, 64, -k_splits);
  return (kb + two - 1) / two <= (kb + one - 1) / one;
}
// The rule for weight gradients with k_splits as aeris_gemm_auto takes it, on a device of `sms` multiprocessors.
extern "C" int aeris_wgrad_takes_pairs(int M, int N, int K, int k_splits, int sms) {
  return N % (G2_BN / 2) == 0 && pairs_pay(M, N, K, EPI_ACC_F32) && slices_stay(M, N, K, k_splits, sms);
}
extern "C" int aeris_gemm_takes_pairs(int M, int N, int K, int epi, int allow_2cta) {
  const bool taken = N % (epi == EPI_SWIGLU || epi == EPI_SWIGLU_BOTH ? G2_BN : G2_BN / 2) == 0;
  return taken && (allow_2cta == 2 || (allow_2cta && pairs_pay(M, N, K, epi)));
}

extern "C" int aeris_gemm_auto(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                               int a_mn, int b_mn, int epi, const void* resid, int ldr, const float* gate,
                               int rows_per_gate, int ld_gate, void* aux, int ld_aux, int swiglu_f, int k_splits,
                               int bn, int allow_2cta, int* status, void* stream) {
  if (allow_2cta == 1 && epi == EPI_ACC_F32 ? aeris_wgrad_takes_pairs(M, N, K, k_splits, num_sms())
                                            : aeris_gemm_takes_pairs(M, N, K, epi, allow_2cta))
    return gemm_two_cta(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, epi, resid, ldr, gate, rows_per_gate, ld_gate, aux,
                        ld_aux, swiglu_f, k_splits, status, stream);
  // few tiles: the smaller ones (wide tiles are for SwiGLU, whose columns come in pairs)
  if (allow_2cta && bn == 0 && (epi == EPI_STORE || epi == EPI_GATE_RESID || epi == EPI_STORE_F32)) bn = 128;
  return gemm_one_cta(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, epi, resid, ldr, gate, rows_per_gate, ld_gate, aux,
                      ld_aux, swiglu_f, k_splits, bn, status, stream);
}

// QKV (or dO) projection whose epilogue performs the Ulysses head<->sequence exchange: C is not written locally;
// every head's tile goes straight into the symmetric buffer of the rank that owns the head (`peers[owner]`).
// A: [M, K] row-major tokens (M = windows * n_local), B: [N, K] weights (or stored [K, N] with b_mn).
extern "C" int aeris_gemm_scatter_heads(const void* A, const void* B, int M, int N, int K, int lda, int ldb,
                                        int b_mn, const void* const* peers, int sp, int sp_rank, int n_local, int L,
                                        int sec_w, int* status, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (M <= 0 || N % G2_BN != 0 || K <= 0 || sp < 1 || sp > 8) return -1;
  if (sec_w % sp != 0 || (sec_w / sp) % 32 != 0 || N % sec_w != 0 || M % n_local != 0) return -2;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.epi = EPI_SCATTER_HEADS; p.C = nullptr; p.ldc = 0;
  p.rows_per_gate = M; p.k_splits = 1; p.status = status;
  p.b_tile_stride = G2_BN; p.b_half_off = G2_BN / 2;
  for (int i = 0; i < sp; ++i) p.scat_peers[i] = const_cast<void*>(peers[i]);
  p.scat_rank = sp_rank; p.scat_n_local = n_local; p.scat_L = L; p.scat_sec_w = sec_w; p.scat_own_w = sec_w / sp;
  p.scat_ld = (N / sec_w) * (sec_w / sp);
  CUtensorMap ta, tb;
  int r = make_tmap_2d_bf16(&ta, A, K, M, lda, G2_BK, G2_BM);
  if (r) return r;
  r = b_mn ? make_tmap_2d_bf16(&tb, B, N, K, ldb, 64, G2_BK) : make_tmap_2d_bf16(&tb, B, K, N, ldb, G2_BK, G2_BN / 2);
  if (r) return r - 100;
  return b_mn ? launch_gemm2<0, 1, 4>(ta, tb, p, stream) : launch_gemm2<0, 0, 4>(ta, tb, p, stream);
}

// GEMM -> reduce-scatter by rows in one kernel: rank `rank` computes its partial product for all `world *
// rows_per_rank` rows (A: [M, K] with K this rank's slice of the reduction dimension) and the epilogue stores each bf16
// tile into slot `rank` of the owner's [world * rows_per_rank, N] buffer `peers[owner]` (peer memory), so the
// transfer rides along tile by tile. The owner sums its `world` slots afterwards (aeris_rs_finalize).
extern "C" int aeris_gemm_rs_push(const void* A, const void* B, int M, int N, int K, int lda, int ldb, int b_mn,
                                  const void* const* peers, int world, int rank, int rows_per_rank, int ld_dst,
                                  int* status, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (M <= 0 || N % G2_BN != 0 || K <= 0 || world < 1 || world > 8 || rank < 0 || rank >= world) return -1;
  if (M != world * rows_per_rank || ld_dst % 8 != 0 || ld_dst < N) return -2;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.epi = EPI_RS_PUSH; p.C = nullptr; p.ldc = 0;
  p.rows_per_gate = M; p.k_splits = 1; p.status = status;
  p.b_tile_stride = G2_BN; p.b_half_off = G2_BN / 2;
  for (int i = 0; i < world; ++i) p.scat_peers[i] = const_cast<void*>(peers[i]);
  p.scat_rank = rank; p.scat_n_local = rows_per_rank; p.scat_ld = ld_dst;
  p.tm_rot = static_cast<int>((static_cast<long long>((rank + 1) % world) * rows_per_rank) / (2 * G2_BM));
  CUtensorMap ta, tb;
  int r = make_tmap_2d_bf16(&ta, A, K, M, lda, G2_BK, G2_BM);
  if (r) return r;
  r = b_mn ? make_tmap_2d_bf16(&tb, B, N, K, ldb, 64, G2_BK) : make_tmap_2d_bf16(&tb, B, K, N, ldb, G2_BK, G2_BN / 2);
  if (r) return r - 100;
  return b_mn ? launch_gemm2<0, 1, 4>(ta, tb, p, stream) : launch_gemm2<0, 0, 4>(ta, tb, p, stream);
}

// All-gather -> GEMM in one kernel (two-CTA tiles). `A` is this rank's [world * rows_per_rank, K] buffer (row pitch K)
// whose chunk `rank` is filled; `peers[p]` is rank p's buffer of the same layout and `counter_peers[p]` its array of 8
// arrival words (peer memory; zero before the first call, never reset). `call_index` counts the calls made on this
// exchange (1, 2, ...; the same on every rank). On return of the kernel the whole gathered A is resident in `A` (the
// weight-gradient product reuses it). The caller synchronises the ranks before the call (every rank is done with the
// previous contents of the buffers). Epilogues: EPI_STORE, EPI_SWIGLU, EPI_SWIGLU_BOTH, EPI_SWIGLU_BWD.
extern "C" int aeris_gemm_allgather_a(void* A, const void* const* peers, const void* const* counter_peers, int world,
                                      int rank, int rows_per_rank, unsigned call_index, const void* B, void* C, int N,
                                      int K, int ldb, int ldc, int b_mn, int epi, const void* resid, int ldr, void* aux,
                                      int ld_aux, int swiglu_f, int* status, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (world < 1 || world > 8 || rank < 0 || rank >= world || rows_per_rank <= 0 || N <= 0 || K <= 0) return -1;
  if (N % G2_BN != 0 || K % 8 != 0 || (static_cast<long long>(rows_per_rank) * K) % 8 != 0) return -2;
  const bool swiglu_fwd = (epi == EPI_SWIGLU || epi == EPI_SWIGLU_BOTH);
  if (swiglu_fwd && b_mn) return -3;
  if (epi != EPI_STORE && !swiglu_fwd && epi != EPI_SWIGLU_BWD) return -4;
  const int M = world * rows_per_rank;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K; p.epi = epi; p.C = C; p.ldc = ldc;
  p.resid = reinterpret_cast<const __nv_bfloat16*>(resid); p.ldr = ldr;
  p.rows_per_gate = M; p.aux = reinterpret_cast<__nv_bfloat16*>(aux); p.ld_aux = ld_aux;
  p.k_splits = 1; p.status = status; p.swiglu_f = swiglu_f;
  if (swiglu_fwd) { p.b_tile_stride = G2_BN / 2; p.b_half_off = swiglu_f; }
  else            { p.b_tile_stride = G2_BN;     p.b_half_off = G2_BN / 2; }
  for (int i = 0; i < world; ++i) {
    p.ag_peers[i] = const_cast<void*>(peers[i]);
    p.ag_count_peers[i] = reinterpret_cast<unsigned*>(const_cast<void*>(counter_peers[i]));
  }
  p.ag_local = A; p.ag_count = p.ag_count_peers[rank]; p.ag_world = world; p.ag_rank = rank; p.ag_rows = rows_per_rank;
  p.ag_expect = call_index;     // multiplied by the grid size at launch
  CUtensorMap ta, tb;
  int r = make_tmap_2d_bf16(&ta, A, K, M, K, G2_BK, G2_BM);
  if (r) return r;
  if (!b_mn) {
    const uint64_t brows = swiglu_fwd ? static_cast<uint64_t>(2) * swiglu_f : static_cast<uint64_t>(N);
    r = make_tmap_2d_bf16(&tb, B, K, brows, ldb, G2_BK, G2_BN / 2);
  } else {
    r = make_tmap_2d_bf16(&tb, B, N, K, ldb, 64, G2_BK);
  }
  if (r) return r - 100;
  return b_mn ? launch_gemm2<0, 1, 4, true>(ta, tb, p, stream) : launch_gemm2<0, 0, 4, true>(ta, tb, p, stream);
}
