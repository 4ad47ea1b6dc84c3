// One cached token through one layer (hawk/hawk.py:206-236 with :164-203 and :61-86), or through the final norm and the
// head (:300-303), as one chain of seven (two) launches for batches of up to 256 rows:
//   norm(residual + branch) | input projection | conv + gates + RG-LRU + gelu(y)*h | output projection |
//   norm(residual + branch) | gate/up projection + gelu(gate)*up | down projection
// or of five (one) for the fewest, which compute the norms inside the projections.  The model uses the chain for up to 32 (bf16
// weights) or 64 (fp32) rows, where it is the faster one; for more it calls its modules, and only direct callers of the
// entry points reach what is here for 65 to 256 rows (6 layers of 2048 in bf16, us: 448 / 690 at 128 / 256 against 346 / 391).
//
// What bounds it: every weight is read once per token, 2.7 GB for the 1.35 B model (0.41 ms at 6.65 TB/s), in launches of
// 1 to 50 MB each, i.e. 1.3 to 8 us of reading against 2 to 3 us in which a launch drains, the next one starts and its
// first loads travel.  So the launches of a chain overlap: each is a programmatic dependent launch, and a projection has
// its shared-memory ring full of weights (which no kernel of the chain writes) before it waits for its predecessor.
#include <algorithm>

#include "decode.cuh"
#include "tc05.cuh"

namespace hawk {
using namespace tc;

// ---------------------------------------------------------------------------------------------
// y[M, N] = x[M, K] . W[N, K]^T for few rows of x (M <= 256): tcgen05 with the roles turned round, 128 rows of W as the
// M side and the tokens as the N side, so that no tensor work is done for padding beyond a multiple of 16 tokens.
//
// A CTA computes 128 rows of W against a slice of K; the `splits` CTAs of a cluster share a tile and add their partial
// sums through each other's shared memory in a fixed order (no workspace, no second launch).  The split is what puts a
// 2048 x 2048 projection (16 tiles) on all SMs; linear_plan() chooses it.  Two or three CTAs fit an SM (rings of 2 to 4
// stages of 64 K; 256 TMEM columns at most), so that the next launch's CTAs load while this one's finish.
//
// WF32: W is fp32 (a model under autocast) and is rounded to bf16 on its way to shared memory by eight warps, the same
// rounding that a cast pass makes: 4 bytes of traffic per weight instead of 4 + 2 + 2.
// GEGLU: W is [gate | up] (2N rows); a tile is 64 gate rows and their 64 up rows and leaves as gelu(gate) * up.
//
// Bound by latency and, past 64 tokens, by the partial sums.  16 tokens, back to back over cold weights: 4096 x 2048 7.0 us
// (8.8 without reading weights early), 2048 x 2048 6.1 (6.8), 2 x 6144 x 2048 with GEGLU 18.7 (20.7), 2048 x 6144 9.6 (10.8),
// where reading takes 2.5, 1.3, 7.6 and 3.8; of the first, 3.4 us pass between the predecessor's end and the last MMA and 1.8
// in the cluster's two barriers, the sums and the store.
// ---------------------------------------------------------------------------------------------
constexpr int DL_ROWS = 128, DL_BK = 64, DL_W_BYTES = DL_ROWS * DL_BK * 2, DL_MAX_STAGES = 6, DL_MAX_SPLITS = 8;
// Bytes of a CTA's ring.  Up to 64 tokens three CTAs fit an SM, so that the next launch's are there to read its weights early
// (16 / 64 tokens through 6 layers of 2048: 308 / 353 us against 337 / 378 with rings of 108 KB, of which two fit); more
// tokens need the larger ring for two stages or three (128 tokens: 448 against 505).
constexpr int dl_ring(int npad) { return npad <= 64 ? 74 * 1024 : 108 * 1024; }

struct LinearArgs {
  int M, N, K, npad, splits, stages, chunk, early;
  const float* wf;   // WF32
  __nv_bfloat16* out;
  int* status;
};

template <bool WF32, bool GEGLU>
__global__ void __launch_bounds__(WF32 ? 320 : 192, 2)
decode_linear_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, LinearArgs p) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[DL_MAX_STAGES], empty_bar[DL_MAX_STAGES], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  const int S = p.splits, rank = S > 1 ? (int)cluster_rank() : 0, tile = blockIdx.x / S;
  const int kblocks = (p.K + DL_BK - 1) / DL_BK, per = (kblocks + S - 1) / S;
  const int kb0 = rank * per, nkb = min(kblocks, kb0 + per) - kb0;  // >= 1: linear_plan()
  const int x_bytes = p.npad * DL_BK * 2, stage_bytes = DL_W_BYTES + x_bytes;
  const int row_lo = GEGLU ? tile * 64 : tile * DL_ROWS, row_hi = GEGLU ? p.N + tile * 64 : row_lo + 64;
  uint32_t tmem_cols = 32;
  while ((int)tmem_cols < p.npad) tmem_cols <<= 1;

  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(&full_bar[s], WF32 ? 9 : 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&done_bar, 1);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(&tmem_slot, tmem_cols);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int* abortp = &abort_flag;

  if (warp == 0) {
    if (lane == 0) {  // ---- TMA producer ----
      auto load_w = [&](int i, int s) {
        unsigned char* st = smem + s * stage_bytes;
        mbar_arrive_expect_tx(&full_bar[s], WF32 ? x_bytes : stage_bytes);
        if (!WF32) {
          tma_load_2d(st, &map_w, &full_bar[s], (kb0 + i) * DL_BK, row_lo);
          tma_load_2d(st + DL_W_BYTES / 2, &map_w, &full_bar[s], (kb0 + i) * DL_BK, row_hi);
        }
      };
      auto load_x = [&](int i, int s) {
        tma_load_2d(smem + s * stage_bytes + DL_W_BYTES, &map_x, &full_bar[s], (kb0 + i) * DL_BK, 0);
      };
      const int pre = min(p.stages, nkb);
      if (p.early)
        for (int i = 0; i < pre; ++i) load_w(i, i);
      pdl_wait();
      pdl_trigger();
      if (!p.early)
        for (int i = 0; i < pre; ++i) load_w(i, i);
      for (int i = 0; i < pre; ++i) load_x(i, i);
      int i = pre;
      for (; i < nkb; ++i) {
        const int s = i % p.stages;
        if (!mbar_wait(&empty_bar[s], ((i / p.stages) & 1) ^ 1, abortp)) break;
        load_w(i, s);
        load_x(i, s);
      }
      if (*abortp) drain_stages(full_bar, p.stages, i);
    }
  } else if (warp == 1) {
    if (lane == 0) {  // ---- MMA issuer ----
      const uint32_t idesc = umma_idesc(DL_ROWS, p.npad);
      int i = 0;
      for (; i < nkb; ++i) {
        const int s = i % p.stages;
        if (!mbar_wait(&full_bar[s], (i / p.stages) & 1, abortp)) break;
        fence_after();
        const uint32_t wa = smem_u32(smem + s * stage_bytes), xa = wa + DL_W_BYTES;
#pragma unroll
        for (int k = 0; k < DL_BK / 16; ++k)
          umma_bf16(tmem, umma_desc_sw128(wa + k * 32), umma_desc_sw128(xa + k * 32), idesc, (i > 0 || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[s]);
      }
      umma_commit(&done_bar);
    }
  } else if (WF32) {  // ---- warps 2-9: W from fp32 to the swizzled bf16 tile ----
    const int t = threadIdx.x - 64;
    float4 v[4][2];  // the thread's four runs of 8 weights of one stage
    auto fetch = [&](int i) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int id = t + q * 256, row = id >> 3, k = (kb0 + i) * DL_BK + (id & 7) * 8;
        const int grow = row < 64 ? row_lo + row : row_hi + row - 64;
        v[q][0] = v[q][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (grow < (GEGLU ? 2 * p.N : p.N) && k < p.K) {
          const float4* src = reinterpret_cast<const float4*>(p.wf + (size_t)grow * p.K + k);
          v[q][0] = src[0];
          v[q][1] = src[1];
        }
      }
    };
    if (!p.early) pdl_wait();
    fetch(0);
    for (int i = 0; i < nkb; ++i) {
      const int s = i % p.stages;
      if (!mbar_wait_warp(&empty_bar[s], ((i / p.stages) & 1) ^ 1, abortp)) break;
      unsigned char* st = smem + s * stage_bytes;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int id = t + q * 256, row = id >> 3, c = id & 7;
        *reinterpret_cast<uint4*>(st + row * 128 + ((c ^ (row & 7)) * 16)) =
            make_uint4(pack_bf16x2(v[q][0].x, v[q][0].y), pack_bf16x2(v[q][0].z, v[q][0].w),
                       pack_bf16x2(v[q][1].x, v[q][1].y), pack_bf16x2(v[q][1].z, v[q][1].w));
      }
      if (i + 1 < nkb) fetch(i + 1);
      fence_smem_to_tma();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[s]);
    }
  }
  __syncwarp();
  pdl_wait();  // every thread that writes results: nothing before this kernel may still be reading that memory

  // ---- epilogue: partial sums to shared memory [tokens][128 rows], added over the cluster, `chunk` tokens at a time ----
  float* part = reinterpret_cast<float*>(smem);  // the ring: every stage has been read once done_bar completes
  const bool writer = warp >= 2 && warp < 6;
  const int quarter = warp & 3;
  bool good = true;
  if (writer) {
    good = mbar_wait_warp(&done_bar, 0, abortp) && !*abortp;
    fence_after();
  }
  for (int t0 = 0; t0 < p.npad; t0 += p.chunk) {
    const int nt = min(p.chunk, p.npad - t0);
    if (writer) {
      for (int c = 0; c < nt; c += 16) {
        uint32_t r[16];
        tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(t0 + c), r);
#pragma unroll
        for (int j = 0; j < 16; ++j)  // a wait that gave up shows in the result
          part[(c + j) * DL_ROWS + quarter * 32 + lane] = good ? __uint_as_float(r[j]) : __int_as_float(0x7fc00000);
      }
    }
    if (S > 1) cluster_sync(); else __syncthreads();
    const int share = (nt + S - 1) / S, first = rank * share, last = min(min(nt, first + share), p.M - t0);
    for (int tok = first + warp; tok < last; tok += nwarps) {
      // all partials of the lane's four columns are requested before any is used: a remote load takes about half a
      // microsecond, and added one by one they were the longest part of the kernel
      const float* mine = part + tok * DL_ROWS + lane * 4;
      float4 b[DL_MAX_SPLITS];
      if (S == 1) {
        b[0] = *reinterpret_cast<const float4*>(mine);
      } else {
#pragma unroll
        for (int s = 0; s < DL_MAX_SPLITS; ++s)
          if (s < S)
            asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
                         : "=f"(b[s].x), "=f"(b[s].y), "=f"(b[s].z), "=f"(b[s].w)
                         : "r"(map_to_rank(mine, (uint32_t)s))
                         : "memory");
      }
      float4 a = b[0];
#pragma unroll
      for (int s = 1; s < DL_MAX_SPLITS; ++s)
        if (s < S) {
          a.x += b[s].x; a.y += b[s].y; a.z += b[s].z; a.w += b[s].w;
        }
      uint2 o = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
      int col = tile * DL_ROWS + lane * 4;
      if (GEGLU) {  // lanes 0-15 hold gate rows, lanes 16-31 the up rows of the same columns; both rounded as projections are
        const uint32_t u0 = __shfl_down_sync(0xffffffffu, o.x, 16), u1 = __shfl_down_sync(0xffffffffu, o.y, 16);
        float2 phi, g0, g1;
        gelu_pair_fast(unpack_bf16x2(o.x), phi, g0);
        gelu_pair_fast(unpack_bf16x2(o.y), phi, g1);
        const float2 v0 = mul2(g0, unpack_bf16x2(u0)), v1 = mul2(g1, unpack_bf16x2(u1));
        o = make_uint2(pack_bf16x2(v0.x, v0.y), pack_bf16x2(v1.x, v1.y));
        col = lane < 16 ? tile * 64 + lane * 4 : p.N;
      }
      if (col < p.N) *reinterpret_cast<uint2*>(p.out + (size_t)(t0 + tok) * p.N + col) = o;
    }
    __syncwarp();
    if (S > 1) cluster_sync(); else __syncthreads();  // the sums have been read before they are overwritten or go away
  }
  fence_before();
  __syncthreads();
  if (abort_flag && threadIdx.x == 0) atomicExch(p.status, 1);
  if (warp == 1) {
    fence_after();
    tmem_dealloc(tmem, tmem_cols);
  }
}

// K splits of a projection: the time of a launch goes with the K blocks that the busiest SM works through, plus about
// 1.5 blocks' worth for adding partial sums, plus 4 for every further wave of the 2 CTAs per SM.
static int linear_plan(int tiles, int kblocks) {
  int best = 1;
  double best_cost = 0;
  const int sms = sm_count();
  for (int s = 1; s <= DL_MAX_SPLITS && s <= kblocks; ++s) {
    const int per = (kblocks + s - 1) / s;
    if ((s - 1) * per >= kblocks) continue;
    const long long ctas = (long long)tiles * s;
    const double cost = (double)((ctas + sms - 1) / sms) * per + (s > 1 ? 1.5 : 0.0) + 4.0 * (double)((ctas - 1) / (2 * sms));
    if (best_cost == 0 || cost < best_cost) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}

static int linear_launch(const __nv_bfloat16* x, const void* w, int w_dtype, __nv_bfloat16* out, int M, int N, int K, bool geglu,
                         bool early, bool pdl, int* status, cudaStream_t st) {
  const int rows = geglu ? 2 * N : N;
  CUtensorMap mx, mw;
  LinearArgs a{};
  a.npad = (M + 15) / 16 * 16;
  if (!make_map_bf16(&mx, x, M, K, K, a.npad)) return HAWK_ERR_DEVICE;
  if (w_dtype == HAWK_BF16) {
    if (!make_map_bf16(&mw, w, rows, K, K, 64)) return HAWK_ERR_DEVICE;
  } else {
    mw = mx;
    a.wf = static_cast<const float*>(w);
  }
  const int stage = DL_W_BYTES + a.npad * DL_BK * 2;
  a.M = M; a.N = N; a.K = K; a.early = early; a.out = out; a.status = status;
  a.stages = std::min(DL_MAX_STAGES, dl_ring(a.npad) / stage);
  const int max_chunk = a.stages * stage / (DL_ROWS * 4) / 16 * 16, chunks = (a.npad + max_chunk - 1) / max_chunk;
  a.chunk = ((a.npad + chunks - 1) / chunks + 15) / 16 * 16;
  const int tiles = geglu ? (N + 63) / 64 : (N + DL_ROWS - 1) / DL_ROWS;
  a.splits = linear_plan(tiles, (K + DL_BK - 1) / DL_BK);
  const int smem = a.stages * stage + 1024;
  auto go = [&](auto kern, unsigned threads) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) {
      (void)cudaGetLastError();
      return (int)HAWK_ERR_LAUNCH;
    }
    return launch_kernel(kern, dim3((unsigned)(tiles * a.splits)), dim3(threads), (size_t)smem, st, pdl, (unsigned)a.splits, mx, mw, a);
  };
  if (w_dtype == HAWK_BF16) return geglu ? go(decode_linear_kernel<false, true>, 192) : go(decode_linear_kernel<false, false>, 192);
  return geglu ? go(decode_linear_kernel<true, true>, 320) : go(decode_linear_kernel<true, false>, 320);
}

// ---------------------------------------------------------------------------------------------
// The same product for at most 16 tokens, with the norm in front of it folded in: five launches per layer instead of seven,
// and none of the cluster's and TMEM's round trips (a projection of one token spent 3.7 us between its predecessor's end and
// its own, of which the weights, already in shared memory, needed none).
//
// mma.sync m16n8k16 with 16 rows of W as the M side and 8 tokens as the N side: a CTA's eight warps take 16 rows of W at a
// time, each its own slice of K, straight from global memory into fragments.  A fragment's k order is free as long as both
// operands use the same: a lane's 16 bytes (8 consecutive k of one row) serve two MMAs.  The first 16 rows' weights are in
// registers (64 KB per CTA, two CTAs per SM) before the kernel waits for its predecessor, the next ones are requested
// before the current ones' sums leave the CTA.  Bound by the latency from one launch to the next: of a layer of width 2048, 31 us
// for one token where its weights take 15.3, 4 each pass between the two norms' inputs and their results, 4 in the recurrent
// branch's step, 0.6 to 1.7 at each of the five boundaries.  24 layers and the head: 1065 us, 858 with the norm's inputs requested
// at once, 831 with the branch's step as it is now.
//
// NORM: x is the residual (1: bf16, 2: fp32), what is multiplied is norm(x + delta); every CTA computes the statistics of its
// few rows itself, CTA 0 writes x + delta.  GEGLU: 8 gate rows and their 8 up rows.
// ---------------------------------------------------------------------------------------------
struct RowsArgs {
  const void* w;
  const void* x;
  const __nv_bfloat16* delta;
  void* x_out;
  const float* norm_w;
  __nv_bfloat16* out;
  int M, N, K, items, early;
  float eps;
};

template <typename WT>
struct WFrag;  // eight consecutive weights of one row
template <>
struct WFrag<__nv_bfloat16> {
  uint4 v;
  __device__ __forceinline__ void zero() { v = make_uint4(0u, 0u, 0u, 0u); }
  __device__ __forceinline__ void load(const __nv_bfloat16* p) {
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  }
  __device__ __forceinline__ uint4 bf16() const { return v; }
};
template <>
struct WFrag<float> {
  float4 a, b;
  __device__ __forceinline__ void zero() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void load(const float* p) {
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w) : "l"(p));
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w) : "l"(p + 4));
  }
  __device__ __forceinline__ uint4 bf16() const {
    return make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w), pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w));
  }
};

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: groups of 8 tokens; KB: blocks of 32 k per warp and step; WARPS: 8, or 16 where a row of W is so long that eight warps
// would take it in three steps with one CTA per SM
template <typename WT, int NT, int KB, int WARPS, bool GEGLU, int NORM>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS) decode_rows_kernel(RowsArgs p) {
  using bf = __nv_bfloat16;
  using TX = typename std::conditional<NORM == 2, float, bf>::type;  // storage of x
  constexpr int XV = sizeof(TX) / 2;                                  // 16-byte loads per 8 elements of x
  __shared__ float red[2][WARPS][16][8 * NT];
  __shared__ float stat[WARPS][8 * NT];
  extern __shared__ __align__(16) float norm_w[];  // NORM: [K]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
  const int chunks = (p.K + 32 * WARPS * KB - 1) / (32 * WARPS * KB);
  const WT* w = static_cast<const WT*>(p.w);
  const TX* x = static_cast<const TX*>(p.x);
  auto k_of = [&](int c, int j) { return ((c * WARPS + warp) * KB + j) * 32 + tig * 8; };

  WFrag<WT> wf[KB][2];
  auto load_w = [&](int item, int c) {
    const int r0 = GEGLU ? item * 8 + gid : item * 16 + gid, r1 = GEGLU ? p.N + r0 : r0 + 8;
    const bool ok0 = r0 < p.N, ok1 = GEGLU ? ok0 : r1 < p.N;
#pragma unroll
    for (int j = 0; j < KB; ++j) {
      const int k = k_of(c, j);
      if (ok0 && k < p.K) wf[j][0].load(w + (size_t)r0 * p.K + k); else wf[j][0].zero();
      if (ok1 && k < p.K) wf[j][1].load(w + (size_t)r1 * p.K + k); else wf[j][1].zero();
    }
  };
  int item = blockIdx.x;
  if (!p.early) pdl_wait();
  load_w(item, 0);
  pdl_wait();
  pdl_trigger();

  uint4 xf[NT][KB];
  float inv[NT];
  if (NORM) {
    for (int k = threadIdx.x * 4; k < p.K; k += WARPS * 128) copy_async16(norm_w + k, p.norm_w + k);
  }
  // NORM: x + delta of chunk c, as the norm sees it, in x's precision.  All of x and four blocks of delta are requested before
  // any is used (block by block these loads took 6 of the kernel's 8 us).
  uint4 xs[NT][NORM ? KB : 1][XV];
  auto fetch_sum = [&](int c) {
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int j = 0; j < KB; ++j) {
        const int k = k_of(c, j), tok = t * 8 + gid;
        const bool ok = k < p.K && tok < p.M;
#pragma unroll
        for (int h = 0; h < XV; ++h) xs[t][j][h] = ok ? ld_dep16(x + (size_t)tok * p.K + k + h * 4) : make_uint4(0u, 0u, 0u, 0u);
      }
    if (p.delta == nullptr) return;
    constexpr int STEP = KB < 4 ? KB : 4;
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int j0 = 0; j0 < KB; j0 += STEP) {
        uint4 dr[STEP][1];
        const int tok = t * 8 + gid;
#pragma unroll
        for (int j = 0; j < STEP; ++j) {
          const int k = k_of(c, j0 + j);
          dr[j][0] = k < p.K && tok < p.M ? ld_dep16(p.delta + (size_t)tok * p.K + k) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int j = 0; j < STEP; ++j) {
          float v[8], d[8];
          unpack8(xs[t][j0 + j], v);
          unpack8(dr[j], d);
#pragma unroll
          for (int q = 0; q < 8; ++q) v[q] += d[q];
          pack8(v, xs[t][j0 + j]);
        }
      }
  };
  auto normalise = [&](int c) {
#pragma unroll
    for (int j = 0; j < KB; ++j) {
      const int k = k_of(c, j);
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        float v[8];
        unpack8(xs[t][j], v);
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = k < p.K ? (v[q] * inv[t]) * norm_w[k + q] : 0.f;
        uint4 o[1];
        pack8(v, o);
        xf[t][j] = o[0];
      }
    }
  };
  auto load_x = [&](int c) {
    if (NORM) {
      fetch_sum(c);
      normalise(c);
    } else {
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int j = 0; j < KB; ++j) {
          const int k = k_of(c, j), tok = t * 8 + gid;
          xf[t][j] = k < p.K && tok < p.M ? ld_dep16(x + (size_t)tok * p.K + k) : make_uint4(0u, 0u, 0u, 0u);
        }
    }
  };
  if (NORM) {
    float ss[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) ss[t] = 0.f;
    for (int c = 0; c < chunks; ++c) {
      fetch_sum(c);
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int j = 0; j < KB; ++j) {
          const int k = k_of(c, j), tok = t * 8 + gid;
          float v[8];
          unpack8(xs[t][j], v);
          if (p.delta && blockIdx.x == 0 && k < p.K && tok < p.M)
            VecIO<TX, 8>::store(static_cast<TX*>(p.x_out) + (size_t)tok * p.K + k, v);
#pragma unroll
          for (int q = 0; q < 8; ++q) ss[t] = fmaf(v[q], v[q], ss[t]);
        }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      ss[t] += __shfl_xor_sync(0xffffffffu, ss[t], 1);
      ss[t] += __shfl_xor_sync(0xffffffffu, ss[t], 2);
      if (tig == 0) stat[warp][t * 8 + gid] = ss[t];
    }
    copy_async_wait();
    __syncthreads();
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < WARPS; ++k) s += stat[k][t * 8 + gid];
      inv[t] = rsqrtf(s / (float)p.K + p.eps);
    }
    if (chunks > 1) fetch_sum(0);
    normalise(0);
  } else {
    load_x(0);
  }

  int par = 0;
  for (; item < p.items; item += gridDim.x, par ^= 1) {
    float acc[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
    for (int c = 0; c < chunks; ++c) {
#pragma unroll
      for (int j = 0; j < KB; ++j) {
        const uint4 a = wf[j][0].bf16(), b = wf[j][1].bf16();
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          mma_16816(acc[t], a.x, b.x, a.y, b.y, xf[t][j].x, xf[t][j].y);
          mma_16816(acc[t], a.z, b.z, a.w, b.w, xf[t][j].z, xf[t][j].w);
        }
      }
      const bool last = c + 1 == chunks;
      if (!last) load_w(item, c + 1);
      else if (item + (int)gridDim.x < p.items) load_w(item + gridDim.x, 0);
      if (chunks > 1) load_x(last ? 0 : c + 1);
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      *reinterpret_cast<float2*>(&red[par][warp][gid][t * 8 + 2 * tig]) = make_float2(acc[t][0], acc[t][1]);
      *reinterpret_cast<float2*>(&red[par][warp][gid + 8][t * 8 + 2 * tig]) = make_float2(acc[t][2], acc[t][3]);
    }
    __syncthreads();  // one per item: `red` alternates, so what is read here is overwritten only after the next one
    const int i = threadIdx.x;
    if (GEGLU) {
      const int j = i & 7, tok = i >> 3, col = item * 8 + j;
      if (tok < p.M && tok < 8 * NT && col < p.N) {
        float g = 0.f, u = 0.f;
#pragma unroll
        for (int k = 0; k < WARPS; ++k) {
          g += red[par][k][j][tok];
          u += red[par][k][j + 8][tok];
        }
        float2 phi, gl;
        gelu_pair_fast(make_float2(from_float_round<bf>(g), 0.f), phi, gl);  // both rounded as projections are
        p.out[(size_t)tok * p.N + col] = __float2bfloat16(gl.x * from_float_round<bf>(u));
      }
    } else {
      const int r = i & 15, tok = i >> 4, col = item * 16 + r;
      if (tok < p.M && tok < 8 * NT && col < p.N) {
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < WARPS; ++k) s += red[par][k][r][tok];
        p.out[(size_t)tok * p.N + col] = __float2bfloat16(s);
      }
    }
  }
}

// decode_rows_kernel or the tensor-core kernel above: 8 tokens or fewer always; up to 16 where a CTA's registers hold the
// whole of a row of W beside two groups of tokens.  One token through 6 layers of width 2048 and the head (bf16) takes 229 us,
// 316 with the other kernel; 16 tokens through 8 layers of width 512 (fp32 weights) 153 against 252.  16 tokens of width 1024
// and 2048 take 246 and 421 us with their x in shared memory (every CTA reads all of it) against 212 and 310.
static bool few_rows(int M, int width) { return M <= 8 || (M <= 16 && width <= 512); }

// norm: 0 x is bf16 and multiplied as it is; 1 / 2: the residual in bf16 / fp32
static int rows_launch(int norm, const void* x, const void* delta, void* x_out, const float* norm_w, float eps, const void* w,
                       int w_dtype, __nv_bfloat16* out, int M, int N, int K, bool geglu, bool early, cudaStream_t st) {
  RowsArgs a{};
  a.w = w; a.x = x; a.delta = static_cast<const __nv_bfloat16*>(delta); a.x_out = x_out; a.norm_w = norm_w; a.out = out;
  a.M = M; a.N = N; a.K = K; a.eps = eps; a.early = early;
  a.items = geglu ? (N + 7) / 8 : (N + 15) / 16;
  const dim3 grid((unsigned)std::min(a.items, 2 * sm_count()));
  // The widest step that the registers hold (128 per thread: 8 blocks of 32 bf16 weights in two rows are 64 of them), and no
  // wider than the eight warps need for all of K.
  const size_t smem = norm ? (size_t)K * 4 : 0;
#define HAWK_ROWS(WT, NT, KB, WARPS, G, NM) \
  return launch_kernel(decode_rows_kernel<WT, NT, KB, WARPS, G, NM>, grid, dim3(WARPS * 32), smem, st, true, 1, a)
#define HAWK_ROWS_KB(G, NM)                                                        \
  do {                                                                             \
    if (w_dtype == HAWK_BF16) {                                                    \
      if (M > 8) {                                                                 \
        if (K <= 512 || NM == 2) HAWK_ROWS(__nv_bfloat16, 2, 2, 8, G, NM);         \
        HAWK_ROWS(__nv_bfloat16, 2, 4, 8, G, NM);                                  \
      }                                                                            \
      if (K <= 512) HAWK_ROWS(__nv_bfloat16, 1, 2, 8, G, NM);                      \
      if (K <= 1024 || NM == 2) HAWK_ROWS(__nv_bfloat16, 1, 4, 8, G, NM);          \
      if constexpr (NM == 0 && !G)                                                 \
        if (K > 2048 && a.items <= sm_count()) HAWK_ROWS(__nv_bfloat16, 1, 8, 16, G, NM); \
      if constexpr (NM != 2) HAWK_ROWS(__nv_bfloat16, 1, 8, 8, G, NM);             \
    }                                                                              \
    if (M > 8) HAWK_ROWS(float, 2, 2, 8, G, NM);                                   \
    if (K <= 512) HAWK_ROWS(float, 1, 2, 8, G, NM);                                \
    if constexpr (NM == 0 && !G)                                                   \
      if (K > 1024 && a.items <= sm_count()) HAWK_ROWS(float, 1, 4, 16, G, NM);    \
    HAWK_ROWS(float, 1, 4, 8, G, NM);                                              \
  } while (0)
  if (geglu) {
    if (norm == 1) HAWK_ROWS_KB(true, 1);
    if (norm == 2) HAWK_ROWS_KB(true, 2);
    return HAWK_ERR_UNSUPPORTED;
  }
  if (norm == 1) HAWK_ROWS_KB(false, 1);
  if (norm == 2) HAWK_ROWS_KB(false, 2);
  HAWK_ROWS_KB(false, 0);
#undef HAWK_ROWS_KB
#undef HAWK_ROWS
}

// ---------------------------------------------------------------------------------------------
// y = rms_norm(x + delta) * w for a few rows: a CTA per row, 8 columns per thread and step, the row in registers between
// the two uses.  One memory round trip and one block reduction: bound by latency, not by its few KB.
// ---------------------------------------------------------------------------------------------
template <typename TX, int NV>
__global__ void __launch_bounds__(256)
decode_norm_kernel(const TX* x, const __nv_bfloat16* delta, TX* x_out, const float* w, __nv_bfloat16* y, int H, float eps) {
  __shared__ float part[8];
  const size_t row = (size_t)blockIdx.x * H;
  pdl_wait();
  pdl_trigger();
  float v[NV][8], wv[NV][8];
  float ss = 0.f;
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    const int j = (c * blockDim.x + threadIdx.x) * 8;
#pragma unroll
    for (int q = 0; q < 8; ++q) v[c][q] = 0.f;
    if (j < H) {
      load_dep8(x + row + j, v[c]);
      load_dep8(w + j, wv[c]);
      if (delta) {
        float d[8];
        load_dep8(delta + row + j, d);
#pragma unroll
        for (int q = 0; q < 8; ++q) v[c][q] = from_float_round<TX>(v[c][q] + d[q]);  // statistics of the value as stored
        VecIO<TX, 8>::store(x_out + row + j, v[c]);
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) ss = fmaf(v[c][q], v[c][q], ss);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = 0.f;
  for (int k = 0; k < (int)blockDim.x / 32; ++k) ss += part[k];
  const float inv = rsqrtf(ss / (float)H + eps);
#pragma unroll
  for (int c = 0; c < NV; ++c) {
    const int j = (c * blockDim.x + threadIdx.x) * 8;
    if (j < H) {
      float o[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) o[q] = (v[c][q] * inv) * wv[c][q];
      VecIO<__nv_bfloat16, 8>::store(y + row + j, o);
    }
  }
}

static int norm_launch(const void* x, const void* delta, void* x_out, const float* w, __nv_bfloat16* y, int M, int H, float eps,
                       int x_dtype, cudaStream_t st) {
  const unsigned threads = (unsigned)std::min(256, (H / 8 + 31) / 32 * 32);
  auto go = [&](auto kern, auto tag) {
    using TX = decltype(tag);
    return launch_kernel(kern, dim3((unsigned)M), dim3(threads), 0, st, true, 1, static_cast<const TX*>(x),
                         static_cast<const __nv_bfloat16*>(delta), static_cast<TX*>(x_out), w, y, H, eps);
  };
#define HAWK_DEC_NORM(TX)                                                   \
  return H <= 2048 ? go(decode_norm_kernel<TX, 1>, TX{})                     \
                   : H <= 4096 ? go(decode_norm_kernel<TX, 2>, TX{}) : go(decode_norm_kernel<TX, 4>, TX{})
  if (x_dtype == HAWK_F32) HAWK_DEC_NORM(float);
  HAWK_DEC_NORM(__nv_bfloat16);
#undef HAWK_DEC_NORM
}

static size_t up256(size_t v) { return (v + 255) & ~(size_t)255; }

struct LayerScratch {
  size_t normed, xy, branch, mixed, act, res, total;
};
static LayerScratch layer_scratch(int64_t B, int64_t H, int64_t R, int64_t I, int res_dtype) {
  LayerScratch L;
  size_t o = 0;
  L.normed = o; o += up256((size_t)B * H * 2);
  L.xy = o;     o += up256((size_t)B * 2 * R * 2);
  L.branch = o; o += up256((size_t)B * R * 2);
  L.mixed = o;  o += up256((size_t)B * H * 2);
  L.act = o;    o += up256((size_t)B * I * 2);
  L.res = o;    o += up256((size_t)B * H * dtype_size(res_dtype));
  L.total = o;
  return L;
}

}  // namespace hawk

using namespace hawk;
using bf = __nv_bfloat16;

extern "C" size_t hawk_decode_layer_workspace_bytes(int B, int H, int R, int I, int res_dtype) {
  if (B < 1 || H < 1 || R < 1 || I < 1 || !valid_dtype(res_dtype)) return 0;
  return layer_scratch(B, H, R, I, res_dtype).total;
}

extern "C" int hawk_decode_layer(const hawk_decode_layer_args* a, void* stream) {
  HAWK_REQUIRE(a, HAWK_ERR_NULL);
  HAWK_REQUIRE(a->residual && a->norm1_w && a->w_xy && a->conv_w && a->conv_b && a->wx && a->wa && a->bx && a->ba && a->lam &&
                   a->w_res && a->norm2_w && a->w_gu && a->w_down && a->state && a->out_residual && a->out_pending &&
                   a->workspace && a->status && (a->conv_state || a->W == 1),
               HAWK_ERR_NULL);
  HAWK_REQUIRE(valid_dtype(a->res_dtype) && valid_dtype(a->state_dtype) && valid_dtype(a->gate_dtype) &&
                   valid_dtype(a->xy_dtype) && valid_dtype(a->resid_dtype) && valid_dtype(a->gu_dtype) && valid_dtype(a->down_dtype),
               HAWK_ERR_DTYPE);
  HAWK_REQUIRE(a->B >= 1 && a->H >= 8 && a->R >= 8 && a->I >= 8 && a->H % 8 == 0 && a->R % 8 == 0 && a->I % 8 == 0 &&
                   a->block_width >= 1 && a->R % a->block_width == 0,
               HAWK_ERR_SHAPE);
  HAWK_REQUIRE(a->B <= 256 && a->H <= 8192 && a->W >= 1 && a->W <= 4 && a->block_width <= 128, HAWK_ERR_UNSUPPORTED);
  const LayerScratch L = layer_scratch(a->B, a->H, a->R, a->I, a->res_dtype);
  HAWK_REQUIRE(a->workspace_bytes >= L.total, HAWK_ERR_WORKSPACE);
  for (const void* q : {a->residual, a->pending, static_cast<const void*>(a->norm1_w), a->w_xy, a->w_res,
                        static_cast<const void*>(a->norm2_w), a->w_gu, a->w_down, static_cast<const void*>(a->out_residual),
                        static_cast<const void*>(a->out_pending), static_cast<const void*>(a->workspace)})
    HAWK_REQUIRE(aligned(q, 16), HAWK_ERR_ALIGN);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto* ws = static_cast<unsigned char*>(a->workspace);
  auto* normed = reinterpret_cast<bf*>(ws + L.normed);
  auto* xy = reinterpret_cast<bf*>(ws + L.xy);
  auto* branch = reinterpret_cast<bf*>(ws + L.branch);
  auto* mixed = reinterpret_cast<bf*>(ws + L.mixed);
  auto* act = reinterpret_cast<bf*>(ws + L.act);
  const int B = a->B, H = a->H, R = a->R, I = a->I;
  const void* res = a->pending ? static_cast<const void*>(ws + L.res) : a->residual;
  if (few_rows(B, std::max(H, R))) {
    const int norm = a->res_dtype == HAWK_F32 ? 2 : 1;
    int rc = rows_launch(norm, a->residual, a->pending, ws + L.res, a->norm1_w, a->eps1, a->w_xy, a->xy_dtype, xy, B, 2 * R, H, false,
                         a->follows_layer != 0, st);
    if (rc == HAWK_OK)
      rc = block_step(xy, 2 * R, a->conv_state, a->conv_w, a->conv_b, a->wx, a->wa, a->bx, a->ba, a->lam, a->state, branch, B, R,
                      a->block_width, a->W, HAWK_BF16, a->state_dtype, a->gate_dtype, true, st);
    if (rc == HAWK_OK) rc = rows_launch(0, branch, nullptr, nullptr, nullptr, 0.f, a->w_res, a->resid_dtype, mixed, B, H, R, false, true, st);
    if (rc == HAWK_OK)
      rc = rows_launch(norm, res, mixed, a->out_residual, a->norm2_w, a->eps2, a->w_gu, a->gu_dtype, act, B, I, H, true, true, st);
    if (rc == HAWK_OK)
      rc = rows_launch(0, act, nullptr, nullptr, nullptr, 0.f, a->w_down, a->down_dtype, static_cast<bf*>(a->out_pending), B, H, I, false, true,
                       st);
    return rc;
  }
  // The chain's first kernel waits for everything before it and the others start only after that, so weights may be read early
  // from the second kernel on, whatever ran before the chain.
  int rc = norm_launch(a->residual, a->pending, a->pending ? ws + L.res : nullptr, a->norm1_w, normed, B, H, a->eps1, a->res_dtype, st);
  if (rc == HAWK_OK) rc = linear_launch(normed, a->w_xy, a->xy_dtype, xy, B, 2 * R, H, false, true, true, a->status, st);
  if (rc == HAWK_OK)
    rc = block_step(xy, 2 * R, a->conv_state, a->conv_w, a->conv_b, a->wx, a->wa, a->bx, a->ba, a->lam, a->state, branch, B, R,
                    a->block_width, a->W, HAWK_BF16, a->state_dtype, a->gate_dtype, true, st);
  if (rc == HAWK_OK) rc = linear_launch(branch, a->w_res, a->resid_dtype, mixed, B, H, R, false, true, true, a->status, st);
  if (rc == HAWK_OK) rc = norm_launch(res, mixed, a->out_residual, a->norm2_w, normed, B, H, a->eps2, a->res_dtype, st);
  if (rc == HAWK_OK) rc = linear_launch(normed, a->w_gu, a->gu_dtype, act, B, I, H, true, true, true, a->status, st);
  if (rc == HAWK_OK)
    rc = linear_launch(act, a->w_down, a->down_dtype, static_cast<bf*>(a->out_pending), B, H, I, false, true, true, a->status, st);
  return rc;
}

extern "C" int hawk_decode_norm_linear(const void* residual, const void* pending, const float* norm_w, float eps, const void* w,
                                       void* out, void* workspace, size_t workspace_bytes, int B, int H, int N, int res_dtype,
                                       int w_dtype, int follows_layer, int* status, void* stream) {
  HAWK_REQUIRE(residual && norm_w && w && out && workspace && status, HAWK_ERR_NULL);
  HAWK_REQUIRE(valid_dtype(res_dtype) && valid_dtype(w_dtype), HAWK_ERR_DTYPE);
  HAWK_REQUIRE(B >= 1 && H >= 8 && H % 8 == 0 && N >= 8 && N % 8 == 0, HAWK_ERR_SHAPE);
  HAWK_REQUIRE(B <= 256 && H <= 8192, HAWK_ERR_UNSUPPORTED);
  const size_t sum = pending ? up256((size_t)B * H * dtype_size(res_dtype)) : 0, need = up256((size_t)B * H * 2) + sum;
  HAWK_REQUIRE(workspace_bytes >= need, HAWK_ERR_WORKSPACE);
  HAWK_REQUIRE(aligned(residual, 16) && aligned(pending, 16) && aligned(norm_w, 16) && aligned(w, 16) && aligned(out, 16) &&
                   aligned(workspace, 16),
               HAWK_ERR_ALIGN);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  auto* normed = reinterpret_cast<bf*>(static_cast<unsigned char*>(workspace) + sum);
  if (few_rows(B, H))
    return rows_launch(res_dtype == HAWK_F32 ? 2 : 1, residual, pending, workspace, norm_w, eps, w, w_dtype, static_cast<bf*>(out), B, N,
                       H, false, follows_layer != 0, st);
  int rc = norm_launch(residual, pending, pending ? workspace : nullptr, norm_w, normed, B, H, eps, res_dtype, st);
  if (rc == HAWK_OK) rc = linear_launch(normed, w, w_dtype, static_cast<bf*>(out), B, N, H, false, true, true, status, st);
  return rc;
}
