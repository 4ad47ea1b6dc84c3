// Fused linear + cross-entropy: the loss in one call, d act and d weight in a second, replacing
// hawk/fused_cross_entropy.py:11-73 (2048-row chunks, three cuBLAS GEMMs and ~8 passes over
// [chunk, V] fp32 temporaries per chunk).
//
// Loss, all on the caller's stream:
//   1. cast           : fp32 weight [V,H] and act [N,H] -> bf16 copies (bf16 inputs are used in place).
//   2. GEMM + softmax epilogue (tcgen05): logits tile = act @ weight^T accumulated in TMEM; the
//      epilogue rounds it to bf16 (as F.linear does under autocast, fused_cross_entropy.py:28),
//      stores it once, and reduces each row's tile to (max, sum exp) online, 32 columns at a time;
//      it also picks out the label's logit.  No fp32 [N,V] tensor is ever written.
//   3. row reduce     : tile statistics -> log-sum-exp per row, loss = mean(lse - correct) (:37-44,59-64).
//   4. dprobs         : logits -> (softmax - onehot) / N in bf16, in place (:47-52); skipped when no gradient
//                       is wanted.
// Gradients: two GEMMs with a plain epilogue that can multiply by a gradient of the loss,
//      d act = dprobs @ weight (:56), d weight = dprobs^T @ act (:55).  Neither needs a transposed copy: an operand
//      whose contraction index is the row index of its tensor (weight in d act; dprobs and act in d weight) is read
//      as an MN-major tile straight from the row-major tensor.  The first call leaves dprobs and the bf16 operands
//      behind for it.
//
// The GEMM is one kernel: C[M,Nc] = A[M,K] . B[Nc,K]^T, bf16 operands, fp32 accumulation.
// A pair of CTAs (cta_group::2) computes a 256*MH x 256 output tile, K in blocks of 64 (128-byte swizzled rows).  What
// bounds a CTA working alone on 128x256 is operand delivery from L2: 48 KB per 512 clocks of MMA, 96 B/clk/SM; a
// pair shares B: 32 KB per CTA in the same time with MH = 1, 24 KB with MH = 2.
//   MH = 1: two TMEM accumulators, the epilogue overlaps the next tile's MMA: the logits, whose epilogue is long.
//   MH = 2: the two 256-row halves fill TMEM and share each B tile: the gradient GEMMs when K is long enough for the
//           epilogue that nothing overlaps (tensor pipe active at N8192 H2048 V8192: 79 % with MH = 1).
// Warp-specialised:
//   warp 0   : TMA producer of its CTA's halves of A and B (cp.async.bulk.tensor, ring of 5 or 4 stages);
//   warp 1   : owns TMEM (512 columns); in the leader CTA it issues tcgen05.mma for the pair;
//   warps 2-9: epilogue, two warps per TMEM lane quarter (128 columns each), overlapping the next tile's MMA.  The
//      softmax epilogue is ~10 issue slots and one MUFU operation per logit; with four warps it, not the MMA, set the
//      pace at H = 512 (N32752 V32000: 1.73 ms for 1.07e12 flop).  Tiles leave through shared memory as TMA box
//      stores: full 128-byte lines.  (fp32 rows stored 16 bytes per lane ran at 1.5 TB/s: d weight of 777 rows,
//      V31999 H1024, 92 us.)
// Persistent over tiles (grid = 2 * min(tiles, SM count / 2)).  Every mbarrier wait is bounded by a clock
// budget; on expiry the kernel records a status word, drains, frees TMEM and returns.
#include <algorithm>

#include "tc05.cuh"

namespace hawk {
using namespace tc;

constexpr int BM = 256, BN = 256, BK = 64, UMMA_K = 16;  // one tcgen05.mma of the pair covers 256 x 256 x 16
constexpr int HALF_BYTES = 128 * BK * 2;                 // one CTA's half of an operand tile: 128 M or N indices x 64 K
constexpr int EPI_WARPS = 8, EPI_COLS = 128;             // columns of a tile per epilogue warp
constexpr int BOX_BYTES = 32 * 128;                      // store box: 32 rows x 64 bf16 or 32 fp32 columns
template <int MH>
struct GemmCfg {
  static constexpr int STAGES = MH == 1 ? 5 : 4;
  static constexpr int A_BYTES = MH * HALF_BYTES;               // A halves first, then the B half
  static constexpr int STAGE_BYTES = A_BYTES + HALF_BYTES;
  static constexpr int NBOX = MH == 1 ? 2 : 1;                  // store boxes per epilogue warp
  static constexpr int SMEM = STAGES * STAGE_BYTES + EPI_WARPS * NBOX * BOX_BYTES + 1024;  // + slack for 1024-byte alignment
  static constexpr int NACC = MH == 1 ? 2 : 1;
};
constexpr int GEMM_THREADS = 64 + 32 * EPI_WARPS;

enum { EPI_LOGITS = 0, EPI_OUT = 1 };

struct EpiParams {
  int M, Nc;                 // valid rows / columns of C
  int k_per_split;           // K blocks per split (EPI_OUT); a tile index runs over tiles x splits
  // EPI_LOGITS
  float2* stats;             // [column groups of 128, M] (max, sum exp)
  float* correct;            // [M] logit at the label
  const long long* labels;   // [M]
  // EPI_OUT
  int out_bf16;              // the store map's type
  const float* scale;        // device scalar multiplied in; null = 1
};

constexpr int MN_BOX = 64 * 128;  // bytes of one [64 columns x 64 rows] box of an MN-major operand

// tile index -> (m_tile, n_tile): groups of GROUP_M row tiles sweep all column tiles, so the tiles
// in flight share a small set of A and B tiles in L2
constexpr int GROUP_M = 8;
__device__ __forceinline__ void tile_coords(int tile, int m_tiles, int n_tiles, int& mt, int& nt) {
  const int per_group = GROUP_M * n_tiles;
  const int g = tile / per_group;
  const int first = g * GROUP_M;
  const int gm = min(GROUP_M, m_tiles - first);
  const int in = tile - g * per_group;
  mt = first + in % gm;
  nt = in / gm;
}

// one 32-column chunk of logits of one row: round to bf16, fold into the running (max, sum exp), pick the label
template <bool FULL>
__device__ __forceinline__ void softmax_chunk(const uint32_t (&v)[32], int cbase, int Nc, long long label, bool row_ok,
                                              float* correct, uint32_t (&packed)[16], float& run_m, float& run_s) {
  float2 vals[16];
  float cmax = -INFINITY;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    packed[j] = pack_bf16x2(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
    vals[j] = unpack_bf16x2(packed[j]);  // the bf16-rounded logits are THE logits
    if (!FULL) {
      if (cbase + 2 * j >= Nc) vals[j].x = -INFINITY;
      if (cbase + 2 * j + 1 >= Nc) vals[j].y = -INFINITY;
    }
    cmax = fmaxf(cmax, fmaxf(vals[j].x, vals[j].y));
  }
  const float new_m = fmaxf(run_m, cmax);
  const float2 off = f2(-new_m * kLog2e);
  const float err = fmaf(new_m, kLog2e, off.x);  // off's rounding, exactly: every term below carries the factor 2^err
  float2 add = f2(0.f);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float2 t = fma2(vals[j], f2(kLog2e), off);
    t.x = ex2_approx(t.x);
    t.y = ex2_approx(t.y);
    add = add2(add, t);
  }
  run_s = fmaf(run_s, ex2_approx((run_m - new_m) * kLog2e), (add.x + add.y) * fmaf(err, -0.69314718f, 1.f));  // 2^-err
  run_m = new_m;
  if (row_ok && label >= cbase && label < cbase + 32) {
    const int at = (int)(label - cbase);
    float pick = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      if (at == 2 * j) pick = vals[j].x;
      if (at == 2 * j + 1) pick = vals[j].y;
    }
    *correct = pick;
  }
}

// An epilogue warp's store boxes of 32 rows x 128 bytes (lane = row; 16-byte piece index XOR row mod 8, the store's
// swizzle), NBOX of them used in turn; every store is one bulk group of lane 0, so that counting groups tells when a box
// has been read out and may be refilled.
template <int NBOX>
__device__ __forceinline__ void box_reuse(int lane) {
  if (lane == 0) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(NBOX - 1) : "memory");
  __syncwarp();
}
__device__ __forceinline__ void box_put(unsigned char* box, int lane, int piece0, const uint32_t (&p)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    *reinterpret_cast<uint4*>(box + lane * 128 + (((piece0 + q) ^ (lane & 7)) * 16)) =
        make_uint4(p[4 * q], p[4 * q + 1], p[4 * q + 2], p[4 * q + 3]);
}
__device__ __forceinline__ void box_store(const CUtensorMap* map, const unsigned char* box, int lane, int col, int row,
                                          int depth, const EpiParams& ep) {
  fence_smem_to_tma();
  __syncwarp();
  if (lane == 0) {
    if (col < ep.Nc && row < ep.M) tma_store_3d(map, box, col, row, depth);
    bulk_commit();  // an empty group where nothing is stored: the group count stays in step
  }
}

// ---------------------------------------------------------------------------------------------
// the GEMM
// ---------------------------------------------------------------------------------------------
// A_MN / B_MN: the operand is read as an MN-major tile, i.e. straight from a row-major [K, M] (or [K, Nc])
// tensor whose rows are the contraction index; its tensor map then has boxes of [64 columns x 64 rows],
// one box per 64 M/N indices, 8192 bytes apart in the stage.
template <int MODE, int MH, bool A_MN, bool B_MN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GEMM_THREADS, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 const __grid_constant__ CUtensorMap map_c, int K, int m_tiles, int n_tiles, int splits, EpiParams ep,
                 int* status) {
  using Cfg = GemmCfg<MH>;
  constexpr int KSTAGES = Cfg::STAGES, STAGE_BYTES = Cfg::STAGE_BYTES, A_BYTES = Cfg::A_BYTES, NACC = Cfg::NACC;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[KSTAGES], empty_bar[KSTAGES], tfull_bar[2], tempty_bar[2];
  __shared__ uint32_t tmem_base_slot;
  __shared__ int abort_flag;

  constexpr uint32_t kIdescMaj = umma_idesc(BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const int first_tile = blockIdx.x >> 1, tile_stride = gridDim.x >> 1;
  const int tiles = m_tiles * n_tiles, num_tiles = tiles * splits;
  const int kblocks = (K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < KSTAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 2 * EPI_WARPS);
    }
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc_pair(&tmem_base_slot, 512);
  fence_before();
  __syncthreads();
  cluster_sync();  // the peer's barriers are initialised before anything is signalled across
  fence_after();
  const uint32_t tmem_base = tmem_base_slot;
  volatile int* abortp = &abort_flag;

  if (warp == 0) {
    // ---------------- TMA producer (each CTA: its own halves; bytes counted on the leader's barrier) ----------------
    if (lane == 0) {
      uint32_t it = 0;
      for (int tile = first_tile; tile < num_tiles && !*abortp; tile += tile_stride) {
        int mt, nt;
        tile_coords(tile % tiles, m_tiles, n_tiles, mt, nt);
        const int kb0 = (tile / tiles) * ep.k_per_split, kb1 = min(kblocks, kb0 + ep.k_per_split);
        const int m0 = mt * BM * MH + (int)rank * 128, n0 = nt * BN + (int)rank * 128;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % KSTAGES;
          const uint32_t ph = (it / KSTAGES) & 1;
          if (!mbar_wait(&empty_bar[s], ph ^ 1, abortp)) break;
          if (rank == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * STAGE_BYTES);
          const uint32_t bar = map_to_rank(&full_bar[s], 0);
          unsigned char* st = smem + s * STAGE_BYTES;
#pragma unroll
          for (int hh = 0; hh < MH; ++hh) {
            if (A_MN) {
#pragma unroll
              for (int q = 0; q < 2; ++q)
                tma_load_2d_pair(st + hh * HALF_BYTES + q * MN_BOX, &map_a, bar, m0 + hh * BM + q * 64, kb * BK);
            } else {
              tma_load_2d_pair(st + hh * HALF_BYTES, &map_a, bar, kb * BK, m0 + hh * BM);
            }
          }
          if (B_MN) {
#pragma unroll
            for (int q = 0; q < 2; ++q) tma_load_2d_pair(st + A_BYTES + q * MN_BOX, &map_b, bar, n0 + q * 64, kb * BK);
          } else {
            tma_load_2d_pair(st + A_BYTES, &map_b, bar, kb * BK, n0);
          }
        }
      }
      // A wait gave up somewhere: let the copies issued last land before the pair's shared memory goes.  The leader
      // holds the barriers that count them (for both CTAs); the peer waits at the cluster barrier below.
      if (*abortp && rank == 0) drain_stages(full_bar, KSTAGES, it);
      // otherwise see every stage freed: the commits that free them are signals from the leader to this CTA
      for (uint32_t j = it > KSTAGES ? it - KSTAGES : 0; j < it && !*abortp; ++j)
        (void)mbar_wait(&empty_bar[j % KSTAGES], (j / KSTAGES) & 1, abortp);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader only) ----------------
    if (lane == 0 && rank == 0) {
      uint32_t it = 0, tcount = 0;
      for (int tile = first_tile; tile < num_tiles && !*abortp; tile += tile_stride, ++tcount) {
        const int acc = NACC == 2 ? (tcount & 1) : 0;
        const uint32_t aph = NACC == 2 ? ((tcount >> 1) & 1) : (tcount & 1);
        if (!mbar_wait(&tempty_bar[acc], aph ^ 1, abortp)) break;
        fence_after();
        const int kb0 = (tile / tiles) * ep.k_per_split, kb1 = min(kblocks, kb0 + ep.k_per_split);
        const uint32_t d_tmem = tmem_base + acc * BN;
        bool ok = true;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int s = it % KSTAGES;
          const uint32_t ph = (it / KSTAGES) & 1;
          if (!mbar_wait(&full_bar[s], ph, abortp)) { ok = false; break; }
          fence_after();
          const uint32_t a_addr = smem_u32(smem + s * STAGE_BYTES);
          const uint32_t b_addr = a_addr + A_BYTES;
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            // K-major: 16 K-elements further along the 128-byte rows; MN-major: 16 K-rows (2048 bytes) further down
            const uint64_t bd = B_MN ? umma_desc_sw128(b_addr + k * UMMA_K * 128, MN_BOX) : umma_desc_sw128(b_addr + k * UMMA_K * 2);
#pragma unroll
            for (int hh = 0; hh < MH; ++hh) {
              const uint32_t ah = a_addr + hh * HALF_BYTES;
              const uint64_t ad = A_MN ? umma_desc_sw128(ah + k * UMMA_K * 128, MN_BOX) : umma_desc_sw128(ah + k * UMMA_K * 2);
              umma_bf16_pair(d_tmem + hh * BN, ad, bd, kIdescMaj, (kb > kb0 || k > 0) ? 1u : 0u);
            }
          }
          umma_commit_pair(&empty_bar[s]);  // frees the stage in both CTAs once these MMAs have read it
        }
        if (!ok) break;
        umma_commit_pair(&tfull_bar[acc]);  // accumulator complete (each CTA's epilogue waits on its own barrier)
      }
    }
  } else {
    // ---------------- epilogue (warps 2..9) ----------------
    const int quarter = warp & 3;  // TMEM lanes 32*quarter .. +31 are the ones this warp may read
    const int half = (warp - 2) >> 2;
    unsigned char* boxes = smem + KSTAGES * STAGE_BYTES + (warp - 2) * Cfg::NBOX * BOX_BYTES;
    const float scale = (MODE == EPI_OUT && ep.scale) ? *ep.scale : 1.f;
    uint32_t tcount = 0;
    for (int tile = first_tile; tile < num_tiles; tile += tile_stride, ++tcount) {
      if (*abortp) break;
      int mt, nt;
      tile_coords(tile % tiles, m_tiles, n_tiles, mt, nt);
      const int acc = NACC == 2 ? (tcount & 1) : 0;
      if (!mbar_wait_warp(&tfull_bar[acc], NACC == 2 ? ((tcount >> 1) & 1) : (tcount & 1), abortp)) break;  // lane 0 waits: the warp cannot diverge
      fence_after();
      const int col0 = nt * BN + half * EPI_COLS;
#pragma unroll 1
      for (int hh = 0; hh < MH; ++hh) {
      const int row0 = (mt * MH + hh) * BM + (int)rank * 128 + quarter * 32, row = row0 + lane;
      const bool row_ok = row < ep.M;
      const uint32_t taddr0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((acc + hh) * BN + half * EPI_COLS);
      uint32_t v[2][32];
      tmem_ld32_async(taddr0, v[0]);

      if (MODE == EPI_LOGITS) {
        float run_m = -INFINITY, run_s = 0.f;
        const long long label = row_ok ? ep.labels[row] : -1;
#pragma unroll
        for (int c = 0; c < EPI_COLS / 32; ++c) {
          tmem_ld_wait();
          if (c + 1 < EPI_COLS / 32) tmem_ld32_async(taddr0 + (c + 1) * 32, v[(c + 1) & 1]);
          const int cbase = col0 + c * 32;
          uint32_t packed[16];
          if (cbase + 32 <= ep.Nc) {
            softmax_chunk<true>(v[c & 1], cbase, ep.Nc, label, row_ok, ep.correct + (row_ok ? row : 0), packed, run_m, run_s);
          } else if (cbase < ep.Nc) {
            softmax_chunk<false>(v[c & 1], cbase, ep.Nc, label, row_ok, ep.correct + (row_ok ? row : 0), packed, run_m, run_s);
          } else {  // whole chunk past the vocabulary (same for every lane); the store clips it
#pragma unroll
            for (int j = 0; j < 16; ++j) packed[j] = 0u;
          }
          // box c/2 of the warp: 32 rows x 64 columns, 16-byte piece index XOR row mod 8 (the store's swizzle)
          unsigned char* box = boxes + (c >> 1) * BOX_BYTES;
          if ((c & 1) == 0) box_reuse<2>(lane);
          box_put(box, lane, (c & 1) * 4, packed);
          if (c & 1) box_store(&map_c, box, lane, col0 + (c >> 1) * 64, row0, 0, ep);
        }
        if (row_ok && col0 < ep.Nc) ep.stats[(long long)(col0 / EPI_COLS) * ep.M + row] = make_float2(run_m, run_s);
      } else {
        const int split = tile / tiles;
        auto chunk = [&](int c) -> const uint32_t(&)[32] {  // waits for chunk c, requests the next one
          tmem_ld_wait();
          if (c + 1 < EPI_COLS / 32) tmem_ld32_async(taddr0 + (c + 1) * 32, v[(c + 1) & 1]);
          return v[c & 1];
        };
        if (ep.out_bf16) {
#pragma unroll
          for (int c = 0; c < EPI_COLS / 32; ++c) {
            const uint32_t(&w)[32] = chunk(c);
            uint32_t packed[16];
#pragma unroll
            for (int j = 0; j < 16; ++j)
              packed[j] = pack_bf16x2(__uint_as_float(w[2 * j]) * scale, __uint_as_float(w[2 * j + 1]) * scale);
            unsigned char* box = boxes + ((c >> 1) % Cfg::NBOX) * BOX_BYTES;
            if ((c & 1) == 0) box_reuse<Cfg::NBOX>(lane);
            box_put(box, lane, (c & 1) * 4, packed);
            if (c & 1) box_store(&map_c, box, lane, col0 + (c >> 1) * 64, row0, split, ep);
          }
        } else {
#pragma unroll
          for (int c = 0; c < EPI_COLS / 32; ++c) {
            const uint32_t(&w)[32] = chunk(c);
            unsigned char* box = boxes + (c % Cfg::NBOX) * BOX_BYTES;
            box_reuse<Cfg::NBOX>(lane);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              uint32_t scaled[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) scaled[j] = __float_as_uint(__uint_as_float(w[16 * q + j]) * scale);
              box_put(box, lane, q * 4, scaled);
            }
            box_store(&map_c, box, lane, col0 + c * 32, row0, split, ep);
          }
        }
      }
      }  // halves
      fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(map_to_rank(&tempty_bar[acc], 0));
    }
    if (lane == 0) bulk_wait_all();
  }

  // ---------------- teardown ----------------
  __syncwarp();
  fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) atomicExch(status, 1);
  cluster_sync();  // neither CTA's barriers or TMEM go while the other may still signal or accumulate into them
  if (warp == 1) {
    fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------------------
// small kernels around the GEMMs
// ---------------------------------------------------------------------------------------------
// stats [groups, N] -> lse [N]; per-block partial sums of (lse - correct) -> partial [gridDim.x].  A block is 32 rows
// x 8 slices of the column groups (a thread per row walked 125 groups alone: 31 us at N = 32760, 16 warps in flight
// per SM at most; 28 us with 8 slices, 32 MB of statistics).
__global__ void __launch_bounds__(256)
ce_row_reduce_kernel(const float2* __restrict__ stats, const float* __restrict__ correct, float* __restrict__ lse,
                     float* __restrict__ partial, int N, int groups) {
  __shared__ float2 sl[8][32];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int row = blockIdx.x * 32 + lane;
  float m = -INFINITY, s = 0.f;
  if (row < N)
    for (int t = slice; t < groups; t += 8) {
      const float2 st = stats[(long long)t * N + row];
      const float nm = fmaxf(m, st.x);
      s = s * expf(m - nm) + st.y * expf(st.x - nm);
      m = nm;
    }
  sl[slice][lane] = make_float2(m, s);
  __syncthreads();
  if (slice == 0) {
    float contrib = 0.f;
    if (row < N) {
      float mm = -INFINITY;
#pragma unroll
      for (int k = 0; k < 8; ++k) mm = fmaxf(mm, sl[k][lane].x);
      float ss = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) ss += sl[k][lane].y * expf(sl[k][lane].x - mm);  // an unused slice: 0 * exp(-inf)
      const float l = mm + logf(ss);
      lse[row] = l;
      contrib = l - correct[row];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) contrib += __shfl_xor_sync(0xffffffffu, contrib, o);
    if (lane == 0) partial[blockIdx.x] = contrib;
  }
}

__global__ void __launch_bounds__(256)
ce_loss_final_kernel(const float* __restrict__ partial, int n, float inv_n, float* __restrict__ loss,
                     const int* __restrict__ status) {
  __shared__ float red[256];
  float s = 0.f;
  for (int i = threadIdx.x; i < n; i += 256) s += partial[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  // a GEMM that abandoned a wait (this call or an earlier one nobody has looked at) shows in the loss itself
  if (threadIdx.x == 0) *loss = *status != 0 ? __int_as_float(0x7fc00000) : red[0] * inv_n;
}

// A GEMM of this call abandoned a wait: make that visible in the result itself (the loss, or the first element of
// each gradient, becomes NaN), since a training loop may not read the status word for many steps.
__global__ void ce_poison_on_abort_kernel(const int* __restrict__ status, void* a, int a_bf16, void* b, int b_bf16) {
  if (*status == 0) return;
  if (a) { if (a_bf16) *static_cast<__nv_bfloat16*>(a) = __float2bfloat16(__int_as_float(0x7fc00000)); else *static_cast<float*>(a) = __int_as_float(0x7fc00000); }
  if (b) { if (b_bf16) *static_cast<__nv_bfloat16*>(b) = __float2bfloat16(__int_as_float(0x7fc00000)); else *static_cast<float*>(b) = __int_as_float(0x7fc00000); }
}

// out = scale * sum over splits of partial [splits][n], in a fixed order; 4 elements per thread (n % 4 == 0)
template <typename TO>
__global__ void __launch_bounds__(256)
split_sum_kernel(const float* __restrict__ partial, long long n, int splits, const float* __restrict__ scale, TO* __restrict__ out) {
  const long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
  if (i >= n) return;
  float4 a = *reinterpret_cast<const float4*>(partial + i);
  for (int s = 1; s < splits; ++s) {
    const float4 b = *reinterpret_cast<const float4*>(partial + s * n + i);
    a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
  }
  const float g = scale ? *scale : 1.f;
  const float v[4] = {a.x * g, a.y * g, a.z * g, a.w * g};
  VecIO<TO, 4>::store(out + i, v);
}

// logits [N, ldl] bf16 -> dprobs = (exp(logit - lse) - onehot) / N, in place.  One CTA per row, 16 bytes
// per thread per step.
__global__ void __launch_bounds__(256)
ce_dprobs_kernel(__nv_bfloat16* __restrict__ logits, long long ldl, const float* __restrict__ lse,
                 const long long* __restrict__ labels, int N, int V, float inv_n) {
  const int r = blockIdx.x;
  if (r >= N) return;
  __nv_bfloat16* row = logits + (long long)r * ldl;
  const float l = lse[r];
  const long long label = labels[r];
  const int nvec = (ldl % 8 == 0) ? V / 8 : 0;
  for (int jv = threadIdx.x; jv < nvec; jv += blockDim.x) {
    const uint4 raw = *reinterpret_cast<const uint4*>(row + jv * 8);
    const int lab = (int)(label - (long long)jv * 8);  // 0..7 when the label is in this vector
    const uint32_t in[4] = {raw.x, raw.y, raw.z, raw.w};
    uint32_t out[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 f = unpack_bf16x2(in[q]);
      float p0 = __expf(f.x - l), p1 = __expf(f.y - l);
      if (lab == 2 * q) p0 -= 1.f;
      if (lab == 2 * q + 1) p1 -= 1.f;
      out[q] = pack_bf16x2(p0 * inv_n, p1 * inv_n);
    }
    *reinterpret_cast<uint4*>(row + jv * 8) = make_uint4(out[0], out[1], out[2], out[3]);
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += blockDim.x) {
    float p = __expf(__bfloat162float(row[c]) - l);
    if ((long long)c == label) p -= 1.f;
    row[c] = __float2bfloat16(p * inv_n);
  }
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
// C[M, Nc] = A . B^T with bf16 operands.  A K-major operand is a row-major [M, K] (or [Nc, K]) tensor; an
// MN-major operand (A_MN / B_MN) is a row-major [K, M] (or [K, Nc]) tensor.  lda / ldb: row pitches.
template <int MODE, int MH, bool A_MN, bool B_MN>
static int launch_gemm(const __nv_bfloat16* A, long long lda, const __nv_bfloat16* B, long long ldb, void* C, bool c_f32,
                       long long ldc, int M, int Nc, int K, int splits, EpiParams ep, int* status, cudaStream_t st) {
  CUtensorMap ma, mb, mc;
  const bool oka = A_MN ? make_map_bf16(&ma, A, K, M, lda, 64) : make_map_bf16(&ma, A, M, K, lda, 128);
  const bool okb = B_MN ? make_map_bf16(&mb, B, K, Nc, ldb, 64) : make_map_bf16(&mb, B, Nc, K, ldb, 128);
  if (!oka || !okb) return HAWK_ERR_DEVICE;
  if (!make_map_store(&mc, C, c_f32, Nc, M, splits, ldc, (long long)M * ldc)) return HAWK_ERR_DEVICE;
  auto kern = gemm_bf16_kernel<MODE, MH, A_MN, B_MN>;
  constexpr int GEMM_SMEM = GemmCfg<MH>::SMEM;
  // per call: the attribute belongs to the current device's copy of the kernel
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM) != cudaSuccess) {
    (void)cudaGetLastError();
    return HAWK_ERR_LAUNCH;
  }
  const int m_tiles = (M + BM * MH - 1) / (BM * MH), n_tiles = (Nc + BN - 1) / BN, kblocks = (K + BK - 1) / BK;
  ep.M = M;
  ep.Nc = Nc;
  ep.k_per_split = (kblocks + splits - 1) / splits;
  const long long work = (long long)m_tiles * n_tiles * splits;
  const int pairs = (int)std::min<long long>(work, sm_count() / 2);
  kern<<<2 * pairs, GEMM_THREADS, GEMM_SMEM, st>>>(ma, mb, mc, K, m_tiles, n_tiles, splits, ep, status);
  return launch_status();
}

// Tile height (MH) and K splits of a gradient GEMM.  With few output tiles most CTA pairs would idle (d act of 1548
// rows at H = 512: 14 tiles of 256 rows on 74 pairs, 310 us unsplit), so K is split; a K block costs 0.37 us with
// MH = 1 and 0.58 us with MH = 2 (two halves), a tile about 5 and 9 us of fill and epilogue, and splits a pass that
// sums the partials.  No split is left without K blocks.
struct GradPlan {
  int mh, splits;
};
static GradPlan plan_grad(long long M, long long Nc, long long K) {
  const long long kb = (K + BK - 1) / BK, pairs = std::max(1, sm_count() / 2);
  GradPlan best{1, 1};
  double best_us = 0;
  for (int mh = 1; mh <= 2; ++mh) {
    const long long tiles = ((M + BM * mh - 1) / (BM * mh)) * ((Nc + BN - 1) / BN);
    for (int s = 1; s <= 32 && s <= kb; ++s) {
      const long long per = (kb + s - 1) / s;
      if ((s - 1) * per >= kb) continue;
      const double waves = (double)((tiles * s + pairs - 1) / pairs);
      const double sum_us = s > 1 ? 4.0 + 4.0 * (double)M * Nc * (s + 1) / 5.0e6 : 0.0;
      const double us = waves * (mh == 1 ? per * 0.37 + 5.0 : per * 0.58 + 9.0) + sum_us;
      if (best_us == 0 || us < best_us) {
        best = GradPlan{mh, s};
        best_us = us;
      }
    }
  }
  return best;
}

static size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

// What the forward leaves for the backward: dprobs and the bf16 copies of fp32 operands (offsets 256-byte aligned)
struct CeSaved {
  size_t wb, ab, logits, total;
  long long ldV;
};
static CeSaved ce_saved(long long N, long long H, long long V, int w_dtype, int a_dtype) {
  CeSaved L;
  L.ldV = (V + 7) & ~7LL;
  size_t o = 0;
  L.wb = o;      o += w_dtype == HAWK_F32 ? up256((size_t)V * H * 2) : 0;
  L.ab = o;      o += a_dtype == HAWK_F32 ? up256((size_t)N * H * 2) : 0;
  L.logits = o;  o += up256((size_t)N * L.ldV * 2);
  L.total = o;
  return L;
}
// Scratch of one call
struct CeScratch {
  size_t stats, correct, lse, partial, total;
  int groups, n_blocks;
};
static CeScratch ce_fwd_scratch(long long N, long long V) {
  CeScratch L;
  L.groups = (int)((V + EPI_COLS - 1) / EPI_COLS);
  L.n_blocks = (int)((N + 31) / 32);
  size_t o = 0;
  L.stats = o;   o += up256((size_t)L.groups * N * sizeof(float2));
  L.correct = o; o += up256((size_t)N * 4);
  L.lse = o;     o += up256((size_t)N * 4);
  L.partial = o; o += up256((size_t)L.n_blocks * 4);
  L.total = o;
  return L;
}
static size_t ce_bwd_scratch(long long N, long long H, long long V) {  // the two GEMMs run one after the other
  const int sa = plan_grad(N, H, V).splits, sw = plan_grad(V, H, N).splits;
  return std::max(sa > 1 ? up256((size_t)sa * N * H * 4) : 0, sw > 1 ? up256((size_t)sw * V * H * 4) : 0);
}

static int check_ce(int64_t N, int64_t H, int64_t V, int w_dtype, int a_dtype) {
  HAWK_REQUIRE(valid_dtype(w_dtype) && valid_dtype(a_dtype), HAWK_ERR_DTYPE);
  HAWK_REQUIRE(N >= 1 && V >= 2 && H >= 8 && H % 8 == 0, HAWK_ERR_SHAPE);
  HAWK_REQUIRE(N < (1LL << 31) - 512 && V < (1LL << 31) - 512 && H < (1LL << 31) - 512, HAWK_ERR_SHAPE);
  return HAWK_OK;
}

// one gradient GEMM: `out` [M, Nc] in out_dtype, times *scale
template <bool A_MN, bool B_MN>
static int grad_gemm(const __nv_bfloat16* A, long long lda, const __nv_bfloat16* B, long long ldb, void* out, int out_dtype,
                     const float* scale, int M, int Nc, int K, float* scratch, int* status, cudaStream_t st) {
  const GradPlan plan = plan_grad(M, Nc, K);
  const int splits = plan.splits;
  EpiParams ep{};
  void* C = splits > 1 ? scratch : out;
  ep.out_bf16 = splits == 1 && out_dtype == HAWK_BF16;
  ep.scale = splits > 1 ? nullptr : scale;
  int rc = plan.mh == 2
               ? launch_gemm<EPI_OUT, 2, A_MN, B_MN>(A, lda, B, ldb, C, !ep.out_bf16, Nc, M, Nc, K, splits, ep, status, st)
               : launch_gemm<EPI_OUT, 1, A_MN, B_MN>(A, lda, B, ldb, C, !ep.out_bf16, Nc, M, Nc, K, splits, ep, status, st);
  if (rc != HAWK_OK || splits == 1) return rc;
  const long long n = (long long)M * Nc;
  const unsigned blocks = (unsigned)((n / 4 + 255) / 256);
  if (out_dtype == HAWK_BF16)
    split_sum_kernel<<<blocks, 256, 0, st>>>(scratch, n, splits, scale, static_cast<__nv_bfloat16*>(out));
  else
    split_sum_kernel<<<blocks, 256, 0, st>>>(scratch, n, splits, scale, static_cast<float*>(out));
  return launch_status();
}

}  // namespace hawk

using namespace hawk;

extern "C" size_t hawk_linear_ce_saved_bytes(int64_t N, int64_t H, int64_t V, int w_dtype, int a_dtype) {
  if (N < 1 || H < 1 || V < 1) return 0;
  return ce_saved(N, H, V, w_dtype, a_dtype).total;
}

extern "C" size_t hawk_linear_ce_scratch_bytes(int64_t N, int64_t H, int64_t V) {
  if (N < 1 || H < 1 || V < 1) return 0;
  return std::max(ce_fwd_scratch(N, V).total, ce_bwd_scratch(N, H, V));
}

extern "C" size_t hawk_linear_ce_workspace_bytes(int64_t N, int64_t H, int64_t V) {
  if (N < 1 || H < 1 || V < 1) return 0;
  return ce_saved(N, H, V, HAWK_F32, HAWK_F32).total + hawk_linear_ce_scratch_bytes(N, H, V);
}

// one cast per fp32 operand, the logits GEMM and the two reductions, the pass that makes dprobs; then a GEMM and, where K is
// split, a sum for each gradient, and the look at the status word
extern "C" int hawk_linear_ce_kernels(int64_t N, int64_t H, int64_t V, int w_dtype, int a_dtype, int want_dw, int want_da) {
  if (N < 1 || H < 1 || V < 1) return 0;
  int n = (w_dtype == HAWK_F32) + (a_dtype == HAWK_F32) + 3;
  if (want_dw || want_da) n += 2;
  if (want_dw) n += plan_grad(V, H, N).splits > 1 ? 2 : 1;
  if (want_da) n += plan_grad(N, H, V).splits > 1 ? 2 : 1;
  return n;
}

extern "C" int hawk_linear_ce_fwd(const void* weight, const void* act, const int64_t* labels, float* loss, void* saved,
                                  size_t saved_bytes, void* scratch, size_t scratch_bytes, int64_t N, int64_t H, int64_t V,
                                  int w_dtype, int a_dtype, int want_grad, int* status, void* stream) {
  HAWK_REQUIRE(weight && act && labels && loss && status, HAWK_ERR_NULL);
  int rc = check_ce(N, H, V, w_dtype, a_dtype);
  if (rc != HAWK_OK) return rc;
  const CeSaved S = ce_saved(N, H, V, w_dtype, a_dtype);
  const CeScratch L = ce_fwd_scratch(N, V);
  HAWK_REQUIRE(saved && saved_bytes >= S.total && scratch && scratch_bytes >= L.total, HAWK_ERR_WORKSPACE);
  HAWK_REQUIRE(aligned(saved, 256) && aligned(scratch, 256) && aligned(weight, 16) && aligned(act, 16), HAWK_ERR_ALIGN);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto* sv = static_cast<unsigned char*>(saved);
  auto* sc = static_cast<unsigned char*>(scratch);
  auto* logits = reinterpret_cast<__nv_bfloat16*>(sv + S.logits);
  auto* stats = reinterpret_cast<float2*>(sc + L.stats);
  auto* correct = reinterpret_cast<float*>(sc + L.correct);
  auto* lse = reinterpret_cast<float*>(sc + L.lse);
  auto* partial = reinterpret_cast<float*>(sc + L.partial);

  // 1. operands in bf16 (row-major, as given: no transposes)
  const __nv_bfloat16* wb = static_cast<const __nv_bfloat16*>(weight);
  const __nv_bfloat16* ab = static_cast<const __nv_bfloat16*>(act);
  if (w_dtype == HAWK_F32) {
    auto* wcast = reinterpret_cast<__nv_bfloat16*>(sv + S.wb);
    rc = hawk_cast_f32_bf16(static_cast<const float*>(weight), wcast, V * H, stream);
    if (rc != HAWK_OK) return rc;
    wb = wcast;
  }
  if (a_dtype == HAWK_F32) {
    auto* acast = reinterpret_cast<__nv_bfloat16*>(sv + S.ab);
    rc = hawk_cast_f32_bf16(static_cast<const float*>(act), acast, N * H, stream);
    if (rc != HAWK_OK) return rc;
    ab = acast;
  }
  // 2. logits + online softmax statistics.  The label's logit is written by the tile that holds the label;
  // a label outside [0, V) matches no tile, so its slot keeps this NaN pattern and the loss comes out NaN
  // (a label in the padding of the last chunk picks -inf: the loss comes out +inf).
  if (cudaMemsetAsync(correct, 0xFF, (size_t)N * sizeof(float), st) != cudaSuccess) {
    (void)cudaGetLastError();
    return HAWK_ERR_LAUNCH;
  }
  EpiParams ep{};
  ep.stats = stats;
  ep.correct = correct;
  ep.labels = reinterpret_cast<const long long*>(labels);
  rc = launch_gemm<EPI_LOGITS, 1, false, false>(ab, H, wb, H, logits, false, S.ldV, (int)N, (int)V, (int)H, 1, ep, status, st);
  if (rc != HAWK_OK) return rc;
  // 3. log-sum-exp per row and the mean loss
  ce_row_reduce_kernel<<<L.n_blocks, 256, 0, st>>>(stats, correct, lse, partial, (int)N, L.groups);
  ce_loss_final_kernel<<<1, 256, 0, st>>>(partial, L.n_blocks, 1.0f / (float)N, loss, status);
  // 4. dprobs in place
  if (want_grad)
    ce_dprobs_kernel<<<(unsigned)N, 256, 0, st>>>(logits, S.ldV, lse, reinterpret_cast<const long long*>(labels), (int)N,
                                                  (int)V, 1.0f / (float)N);
  return launch_status();
}

extern "C" int hawk_linear_ce_bwd(const void* weight, const void* act, const void* saved, size_t saved_bytes,
                                  const float* grad_loss, void* dweight, int dw_dtype, void* dact, int da_dtype,
                                  void* scratch, size_t scratch_bytes, int64_t N, int64_t H, int64_t V, int w_dtype,
                                  int a_dtype, int* status, void* stream) {
  HAWK_REQUIRE(weight && act && status && (dweight || dact), HAWK_ERR_NULL);
  HAWK_REQUIRE(valid_dtype(dw_dtype) && valid_dtype(da_dtype), HAWK_ERR_DTYPE);
  int rc = check_ce(N, H, V, w_dtype, a_dtype);
  if (rc != HAWK_OK) return rc;
  const CeSaved S = ce_saved(N, H, V, w_dtype, a_dtype);
  HAWK_REQUIRE(saved && saved_bytes >= S.total, HAWK_ERR_WORKSPACE);
  const size_t need = ce_bwd_scratch(N, H, V);
  HAWK_REQUIRE(need == 0 || (scratch && scratch_bytes >= need), HAWK_ERR_WORKSPACE);
  HAWK_REQUIRE(aligned(saved, 256) && aligned(scratch, 16) && aligned(dweight, 16) && aligned(dact, 16) &&
                   aligned(weight, 16) && aligned(act, 16) && aligned(grad_loss, 4),
               HAWK_ERR_ALIGN);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const auto* sv = static_cast<const unsigned char*>(saved);
  const auto* dprobs = reinterpret_cast<const __nv_bfloat16*>(sv + S.logits);
  const auto* wb = static_cast<const __nv_bfloat16*>(w_dtype == HAWK_F32 ? static_cast<const void*>(sv + S.wb) : weight);
  const auto* ab = static_cast<const __nv_bfloat16*>(a_dtype == HAWK_F32 ? static_cast<const void*>(sv + S.ab) : act);
  auto* part = static_cast<float*>(scratch);
  if (dact) {    // d act [N,H] = dprobs [N,V] . W [V,H]   : A K-major (dprobs rows), B MN-major (W's rows are the K index)
    rc = grad_gemm<false, true>(dprobs, S.ldV, wb, H, dact, da_dtype, grad_loss, (int)N, (int)H, (int)V, part, status, st);
    if (rc != HAWK_OK) return rc;
  }
  if (dweight) {  // d weight [V,H] = dprobs^T . act [N,H] : A and B MN-major (the rows of dprobs and act are the K index)
    rc = grad_gemm<true, true>(dprobs, S.ldV, ab, H, dweight, dw_dtype, grad_loss, (int)V, (int)H, (int)N, part, status, st);
    if (rc != HAWK_OK) return rc;
  }
  ce_poison_on_abort_kernel<<<1, 1, 0, st>>>(status, dweight, dw_dtype == HAWK_BF16, dact, da_dtype == HAWK_BF16);
  return launch_status();
}

extern "C" int hawk_linear_ce_fwd_bwd(const void* weight, const void* act, const int64_t* labels, float* loss,
                                      float* dweight, float* dact, void* workspace, size_t workspace_bytes,
                                      int64_t N, int64_t H, int64_t V, int dtype, int* status, void* stream) {
  HAWK_REQUIRE(weight && act && labels && loss && dweight && dact && status, HAWK_ERR_NULL);
  int rc = check_ce(N, H, V, dtype, dtype);
  if (rc != HAWK_OK) return rc;
  const size_t saved = ce_saved(N, H, V, dtype, dtype).total, scratch = hawk_linear_ce_scratch_bytes(N, H, V);
  HAWK_REQUIRE(workspace && workspace_bytes >= hawk_linear_ce_workspace_bytes(N, H, V), HAWK_ERR_WORKSPACE);
  HAWK_REQUIRE(aligned(workspace, 256) && aligned(dweight, 16) && aligned(dact, 16) && aligned(weight, 16) &&
                   aligned(act, 16),
               HAWK_ERR_ALIGN);
  auto* sc = static_cast<unsigned char*>(workspace) + saved;
  rc = hawk_linear_ce_fwd(weight, act, labels, loss, workspace, saved, sc, scratch, N, H, V, dtype, dtype, 1, status, stream);
  if (rc != HAWK_OK) return rc;
  rc = hawk_linear_ce_bwd(weight, act, workspace, saved, nullptr, dweight, HAWK_F32, dact, HAWK_F32, sc, scratch, N, H, V,
                          dtype, dtype, status, stream);
  if (rc != HAWK_OK) return rc;
  ce_poison_on_abort_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(status, loss, 0, nullptr, 0);
  return launch_status();
}
