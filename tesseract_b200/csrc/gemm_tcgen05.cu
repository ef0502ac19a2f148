// bf16 GEMM on the 5th-generation tensor cores: C[M,N] (+)= op(A) * op(B), fp32 accumulation in TMEM.
//
// Persistent, warp-specialised kernel, one CTA per SM:
//   warp 0      TMA producer: cp.async.bulk.tensor tiles of A and B into a 128-byte-swizzled smem ring
//   warp 1      allocates TMEM; one thread issues tcgen05.mma (128 x BN x 16) and tcgen05.commit
//   warps 2-5   epilogue: tcgen05.ld the finished accumulator (double-buffered in TMEM), convert, store
// Operands may be K-major (row-major [rows, K]) or M/N-major (row-major [K, rows]); the second form is
// what the backward GEMMs of a Linear layer need (dX = dY * W, dW = dY^T * X) without any transposes.
//
// Replaces the cuBLASLt bridge of the reference (src/cuda/MatMul.cpp:422-490) for every dense
// Linear forward/backward.
#include "common.cuh"

#include <mutex>
#include <type_traits>
#include <unordered_map>

namespace tsb {
namespace {

constexpr int BM = 128;
constexpr int BK = 64;  // 64 bf16 = one 128-byte swizzle row
constexpr int kGemmThreads = 192;

template <int BN>
struct GemmCfg {
  static constexpr int kStageBytesA = BM * BK * 2;
  static constexpr int kStageBytesB = BN * BK * 2;
  static constexpr int kStageBytes = kStageBytesA + kStageBytesB;
  static constexpr int kStages = (BN >= 256) ? 4 : (BN >= 128 ? 6 : (BN >= 64 ? 8 : 10));
  static constexpr int kSmemBytes = kStages * kStageBytes + 1024;  // + alignment slack
  static constexpr int kTmemCols = (2 * BN < 32) ? 32 : 2 * BN;
};

struct TileCoord {
  int m_blk, n_blk;
};

__device__ __forceinline__ TileCoord tile_coord(int t, int num_m, int num_n, int GM = 16) {
  const int group_size = GM * num_n;
  const int group_id = t / group_size;
  const int first_m = group_id * GM;
  const int gm = min(num_m - first_m, GM);
  const int r = t - group_id * group_size;
  return {first_m + r % gm, r / gm};
}

// Grouped GEMMs (MoE experts) run through the same kernel. `offsets` (device, int32 [groups + 1], every entry a
// multiple of 128, so no 128-row block and no 64-row reduction step straddles two groups) is read by the kernel,
// never by the host:
//   mode 1  rows grouped (expert forward / input gradient): row block m belongs to the group g with
//           offsets[g] <= 128 m < offsets[g + 1]; the B tensor map stacks the groups' matrices and its row
//           coordinate advances by b_group_rows per group; row blocks at or beyond offsets[groups] are skipped.
//   mode 2  reduction grouped (expert weight gradient, A and B both MN-major): work item (g, m_blk, n_blk) reduces
//           over rows [offsets[g], offsets[g + 1]) and writes C + g * c_group_stride; an empty group adds nothing.
//   mode 1 with `row_tags` (expert-parallel return path): the result rows do not go to C but straight to the rank
//           each row came from -- row r with tag t >= 0 is stored at peer_out[t >> 24] + (t & 0xFFFFFF) * ldc (peer-mapped
//           memory of that rank, over NVLink), rows with a negative tag (padding) are dropped. The all-to-all that
//           returns expert results is the epilogue of the down projection; nothing is written locally.
// Without offsets, `inputs` > 0: result columns from col_start[i] on read the i-th of several inputs stacked `a_group_rows` rows apart
// in A (column tiles do not straddle a start).
struct GroupArgs {
  const int* offsets;
  int groups;
  int mode;
  long long b_group_rows;
  long long c_group_stride;
  const int* row_tags = nullptr;
  long long peer_rows = 0;
  void* peer_out[8] = {};
  int act = 0;             // mode 1: 1 = relu(result)^2
  int inputs = 0;
  int a_group_rows = 0;
  int col_start[8] = {};
};

__device__ __forceinline__ int input_row_offset(const GroupArgs& g, int col) {
  int off = 0;
#pragma unroll
  for (int i = 1; i < 8; ++i)
    if (i < g.inputs && col >= g.col_start[i]) off = i * g.a_group_rows;
  return off;
}

__device__ __forceinline__ int group_of_row(const GroupArgs& g, int row) {
  int e = 0;
  while (e + 1 < g.groups && __ldg(g.offsets + e + 1) <= row) ++e;
  return e;
}

// 32 columns of a result row from `col0` on: stored, added to what is there (ACCUM), or, as slices of a split reduction, added with
// fp32 atomics unless the slice is empty.
template <typename OutT, bool ACCUM>
__device__ __forceinline__ void store_columns(OutT* crow, int col0, int N, bool vec_ok, const uint32_t (&r)[32], bool slices, bool empty_slice) {
  if (vec_ok && col0 + 32 <= N) {
    if constexpr (sizeof(OutT) == 2) {
      uint4* dst = reinterpret_cast<uint4*>(crow + col0);
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[v * 8 + j]);
        if constexpr (ACCUM) {
          const uint4 old = dst[v];
          const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&old);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 of = __bfloat1622float2(o2[j]);
            f[2 * j] += of.x;
            f[2 * j + 1] += of.y;
          }
        }
        uint4 o;
        o.x = pack_bf16x2(f[0], f[1]);
        o.y = pack_bf16x2(f[2], f[3]);
        o.z = pack_bf16x2(f[4], f[5]);
        o.w = pack_bf16x2(f[6], f[7]);
        dst[v] = o;
      }
    } else {
      float4* dst = reinterpret_cast<float4*>(crow + col0);
#pragma unroll
      for (int v = 0; v < 8; ++v) {
        float4 o = make_float4(__uint_as_float(r[v * 4]), __uint_as_float(r[v * 4 + 1]), __uint_as_float(r[v * 4 + 2]),
                               __uint_as_float(r[v * 4 + 3]));
        if (slices) {
          if (!empty_slice) atomicAdd(&dst[v], o);
          continue;
        }
        if constexpr (ACCUM) {
          const float4 old = dst[v];
          o.x += old.x;
          o.y += old.y;
          o.z += old.z;
          o.w += old.w;
        }
        dst[v] = o;
      }
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    if (col0 + j < N) {
      float v = __uint_as_float(r[j]);
      if constexpr (sizeof(OutT) == 4) {
        if (slices) {
          if (!empty_slice) atomicAdd(reinterpret_cast<float*>(crow) + col0 + j, v);
          continue;
        }
      }
      if constexpr (ACCUM) v += to_f32<OutT>(crow[col0 + j]);
      crow[col0 + j] = from_f32<OutT>(v);
    }
  }
}

template <int BN, bool A_MN, bool B_MN, typename OutT, bool ACCUM>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, OutT* __restrict__ C,
                 int M, int N, int K, long long ldc, int* status, int split_k, GroupArgs grp) {
  using Cfg = GemmCfg<BN>;
  constexpr int STAGES = Cfg::kStages;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  __shared__ __align__(8) uint64_t full_bar[STAGES];
  __shared__ __align__(8) uint64_t empty_bar[STAGES];
  __shared__ __align__(8) uint64_t tmem_full_bar[2];
  __shared__ __align__(8) uint64_t tmem_empty_bar[2];
  __shared__ uint32_t tmem_base_smem;
  __shared__ volatile int cta_abort;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;

  const int num_m = (M + BM - 1) / BM;
  const int num_n = (N + BN - 1) / BN;
  // split_k > 1: work item t covers K slice (t % split_k) of output tile (t / split_k); slices are summed with
  // fp32 atomics by the epilogue (ATOMIC_OUT instantiation, C zero-initialised by the caller)
  const int gmode = grp.offsets ? grp.mode : 0;
  const int num_tiles = num_m * num_n * (gmode == 2 ? grp.groups : split_k);
  const int total_kb = (K + BK - 1) / BK;
  const int kb_per = (total_kb + split_k - 1) / split_k;
  const int m_limit = (gmode == 1) ? __ldg(grp.offsets + grp.groups) : M;  // mode 1: rows in use
  const int tiles_per_group = num_m * num_n;

  if (threadIdx.x == 0) {
    cta_abort = 0;
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full_bar[a], 1);
      mbar_init(&tmem_empty_bar[a], 4);
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(&tmem_base_smem, Cfg::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    // (The loops of warps 0 and 1 are walked by the whole warp, and one thread issues: see elect_one.)
    const bool lead = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      const TileCoord tc = (gmode == 2) ? tile_coord(t % tiles_per_group, num_m, num_n) : tile_coord(t / split_k, num_m, num_n);
      const int m0 = tc.m_blk * BM;
      const int n0 = tc.n_blk * BN;
      int kb0 = (t % split_k) * kb_per;
      int kb1 = min(total_kb, kb0 + kb_per);
      int b_row_off = 0;  // rows of the stacked B tensor map before this tile's group
      const int a_row = m0 + input_row_offset(grp, n0);
      if (gmode == 1) {
        if (m0 >= m_limit) continue;
        b_row_off = static_cast<int>(group_of_row(grp, m0) * grp.b_group_rows);
      } else if (gmode == 2) {
        const int g = t / tiles_per_group;
        kb0 = __ldg(grp.offsets + g) / BK;
        kb1 = __ldg(grp.offsets + g + 1) / BK;
      }
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        ok = mbar_wait_warp(&empty_bar[stage], phase ^ 1u, &cta_abort, status);
        if (!ok) break;
        uint8_t* sA = smem + stage * Cfg::kStageBytes;
        uint8_t* sB = sA + Cfg::kStageBytesA;
        if (lead) {
          mbar_expect_tx(&full_bar[stage], Cfg::kStageBytes);
          if (!A_MN) {
            tma_load_2d(sA, &tmA, &full_bar[stage], kb * BK, a_row);
          } else {
#pragma unroll
            for (int i = 0; i < BM / 64; ++i) tma_load_2d(sA + i * 8192, &tmA, &full_bar[stage], m0 + i * 64, kb * BK);
          }
          if (!B_MN) {
            tma_load_2d(sB, &tmB, &full_bar[stage], kb * BK, n0 + b_row_off);
          } else {
#pragma unroll
            for (int i = 0; i < BN / 64; ++i)
              tma_load_2d(sB + i * 8192, &tmB, &full_bar[stage], n0 + i * 64, kb * BK + b_row_off);
          }
        }
        __syncwarp();
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok) break;
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    const uint32_t lead = elect_one() ? 1u : 0u;
    constexpr uint32_t idesc = umma_idesc(BM, BN, 1, 1, A_MN ? 1 : 0, B_MN ? 1 : 0);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      int kb0 = (t % split_k) * kb_per;
      int kb1 = min(total_kb, kb0 + kb_per);
      if (gmode == 1) {
        if (tile_coord(t, num_m, num_n).m_blk * BM >= m_limit) continue;
      } else if (gmode == 2) {
        const int g = t / tiles_per_group;
        kb0 = __ldg(grp.offsets + g) / BK;
        kb1 = __ldg(grp.offsets + g + 1) / BK;
      }
      bool ok = mbar_wait_warp(&tmem_empty_bar[acc], acc_phase ^ 1u, &cta_abort, status);
      if (!ok) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * BN);
      for (int kb = kb0; kb < kb1; ++kb) {
        ok = mbar_wait_warp(&full_bar[stage], phase, &cta_abort, status);
        if (!ok) break;
        tc_fence_after();
        const uint32_t a_base = smem_u32(smem + stage * Cfg::kStageBytes);
        const uint32_t b_base = a_base + Cfg::kStageBytesA;
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          const uint64_t adesc = A_MN ? umma_smem_desc_sw128(a_base + k * 2048, 8192, 1024)
                                      : umma_smem_desc_sw128(a_base + k * 32, 16, 1024);
          const uint64_t bdesc = B_MN ? umma_smem_desc_sw128(b_base + k * 2048, 8192, 1024)
                                      : umma_smem_desc_sw128(b_base + k * 32, 16, 1024);
          umma_f16_if(lead, d_tmem, adesc, bdesc, idesc, (kb > kb0 || k != 0) ? 1u : 0u);
        }
        umma_commit_if(lead, &empty_bar[stage]);  // frees the smem stage once these MMAs have read it
        if (++stage == STAGES) {
          stage = 0;
          phase ^= 1u;
        }
      }
      if (!ok) break;
      umma_commit_if(lead, &tmem_full_bar[acc]);  // accumulator complete
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3;  // TMEM lane quadrant this warp may read
    const int row_in_tile = q * 32 + lane;
    const bool vec_ok = (ldc % (16 / sizeof(OutT)) == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      const TileCoord tc = (gmode == 2) ? tile_coord(t % tiles_per_group, num_m, num_n) : tile_coord(t / split_k, num_m, num_n);
      const int m0 = tc.m_blk * BM;
      const int n0 = tc.n_blk * BN;
      bool empty_slice = (t % split_k) * kb_per >= total_kb;
      OutT* Cg = C;
      if (gmode == 1) {
        if (m0 >= m_limit) continue;
      } else if (gmode == 2) {
        const int g = t / tiles_per_group;
        empty_slice = __ldg(grp.offsets + g) >= __ldg(grp.offsets + g + 1);
        Cg = C + static_cast<long long>(g) * grp.c_group_stride;
      }
      if (!mbar_wait(&tmem_full_bar[acc], acc_phase, &cta_abort, status)) break;
      tc_fence_after();
      const int row = m0 + row_in_tile;
      OutT* crow = Cg + static_cast<long long>(row) * ldc;
      bool row_ok = row < M;
      if (gmode == 1 && grp.row_tags) {
        const int tag = row_ok ? __ldg(grp.row_tags + row) : -1;
        const long long slot = tag & 0xFFFFFF;
        row_ok = tag >= 0 && slot < grp.peer_rows;
        if (row_ok) {
          const int owner = (tag >> 24) & 7;
          void* base = grp.peer_out[0];      // selected by comparison: a dynamic index would move the array to local memory
#pragma unroll
          for (int r = 1; r < 8; ++r)
            if (owner == r) base = grp.peer_out[r];
          crow = static_cast<OutT*>(base) + slot * ldc;
        }
      }
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32(tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN + c * 32), r);
        tmem_ld_wait();
        if (gmode == 2 && empty_slice) {  // a group without rows: nothing was accumulated
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
        if (gmode == 1 && grp.act) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float f = fmaxf(__uint_as_float(r[j]), 0.f);
            r[j] = __float_as_uint(f * f);
          }
        }
        const int col0 = n0 + c * 32;
        if (row_ok && col0 < N) {
          store_columns<OutT, ACCUM>(crow, col0, N, vec_ok, r, split_k > 1, empty_slice);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tmem_empty_bar[acc]);
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1u;
    }
  }

  // ------------------------------------------------------------ tear-down
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (cta_abort) {
      // Give copies and MMAs that are still in flight a bounded moment to land before TMEM goes away.
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::kTmemCols);
  }
}

// ---------------------------------------------------------------- two SMs on one tile
// The same product on tiles that a cluster of two CTAs works on together: `tcgen05.mma.cta_group::2`, issued by the first CTA, multiplies
// 256 rows of A (128 in each CTA's shared memory) with n <= 256 columns of B (n / 2 in each), and each CTA's TMEM receives its 128 rows.
// TMEM holds two such accumulators, and they are used in either of two ways:
//   whole tiles   256 x 2 n: each block of A that is staged meets two blocks of B, so that 48 KB come in for what two tiles would need 64 KB
//                 for, and the second product finds A in the tensor core's buffer. What bounds a large product is power, and
//                 bytes moved through the L2 and shared memory cost it. No accumulator is left to work on during the stores; instead the halves of a tile run
//                 apart by as many blocks of K as the ring holds, at its end (the first is stored while the second catches up) and at its start.
//   halves        256 x n, one accumulator after the other: the rest of the tiles where that is at most a round of halves, and products
//                 that have few tiles or are less than 6144 deep (the first half's stores start earlier).
// Rows leave through shared memory and TMA; an accumulated product reads what it adds to while its products are formed.
//   every CTA   warp 0 loads its halves of A and B; the bytes are counted on the first CTA's barrier. Warps 2-5 store its rows.
//   first CTA   warp 1 issues the MMAs; its commits arrive in both CTAs.
// Sustained under the power limit, against tiles of 256 x 256 only, issued by one lane's loop and stored from registers (us):
//   forward          8192 x 28672 x 4096 1489 -> 1327    8192 x 4096 x 14336 790 -> 669     3003 x 2048 x 8192 106 -> 85
//   input gradient   8192 x 4096 x 28672 1575 -> 1306    8192 x 14336 x 4096 796 -> 670     3003 x 2048 x 16384 208 -> 164
//   weight gradient  28672 x 4096 x 8192 1690 -> 1447    128256 x 4096 x 4096 3788 -> 3286  16384 x 2048 x 3003 179 -> 154
// (1310 - 1480 TFLOP/s for the large ones.)
struct PairTile {
  static constexpr int kHalfBytes = 128 * BK * 2;                   // 128 x 64 of an operand
  static constexpr int kRingBytes = 12 * kHalfBytes;                // four stages of A and two of B, or six of A and one of B
  static constexpr int kOutBytes = 32 * 128, kOutBufs = 2;          // a storing warp's pieces of C: 32 rows of 128 bytes
  static constexpr int kSmemBytes = kRingBytes + 4 * kOutBufs * kOutBytes + 1024, kTmemCols = 512;
};

// How C is cut: `num_m` x `num_w` tiles of 256 rows and `per` times `n` columns. Items below `full` are whole tiles, each two after them
// the halves of one.
struct PairPlan {
  int n, per, group, num_m, num_w, full, items;
};
struct PairItem {
  int m0, c0, halves;
};
__device__ __forceinline__ PairItem pair_item(const PairPlan& pl, int t, int N) {
  const int rest = t - pl.full, tile = rest < 0 ? t : pl.full + (rest >> 1);
  const TileCoord tc = tile_coord(tile, pl.num_m, pl.num_w, pl.group);
  const int c0 = (tc.n_blk * pl.per + (rest < 0 ? 0 : rest & 1)) * pl.n;
  const int fit = c0 >= N ? 0 : c0 + pl.n < N ? 2 : 1;
  return {tc.m_blk * 256, c0, min(fit, rest < 0 ? pl.per : 1)};
}

struct RingCursor {
  int stages, stage = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ explicit RingCursor(int n) : stages(n) {}
  __device__ __forceinline__ void next() {
    if (++stage == stages) {
      stage = 0;
      phase ^= 1u;
    }
  }
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Address, in the cluster's window, of the first CTA's copy of a shared variable.
__device__ __forceinline__ uint32_t in_first_cta(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// A copy into this CTA's shared memory whose bytes are counted on a barrier of either CTA of the pair.
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* tmap, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(tmap), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair_if(uint32_t pred, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "setp.ne.b32 q, %5, 0;\n"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(tmem_d),
      "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(pred)
      : "memory");
}
// Two products of the same rows of A, one right behind the other: the first leaves them in the tensor core's buffer, the second takes them
// from there.
__device__ __forceinline__ void umma_f16_pair_twice_if(uint32_t pred, uint32_t tmem_d0, uint32_t tmem_d1, uint64_t desc_a, uint64_t desc_b0,
                                                       uint64_t desc_b1, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.b32 p, %6, 0;\n"
      "setp.ne.b32 q, %7, 0;\n"
      "@q tcgen05.mma.cta_group::2.kind::f16.collector::a::fill [%0], %2, %3, %5, p;\n"
      "@q tcgen05.mma.cta_group::2.kind::f16.collector::a::lastuse [%1], %2, %4, %5, p;\n"
      "}\n" ::"r"(tmem_d0),
      "r"(tmem_d1), "l"(desc_a), "l"(desc_b0), "l"(desc_b1), "r"(idesc), "r"(accumulate), "r"(pred)
      : "memory");
}
// Arrives on the barrier at this offset in both CTAs.
__device__ __forceinline__ void umma_commit_pair_if(uint32_t pred, uint64_t* bar) {
  asm volatile(
      "{\n"
      ".reg .pred q;\n"
      "setp.ne.b32 q, %2, 0;\n"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
      "}\n" ::"r"(smem_u32(bar)),
      "h"(static_cast<uint16_t>(3)), "r"(pred)
      : "memory");
}

template <bool A_MN, bool B_MN, typename OutT, bool ACCUM>
// (At most 168 registers where rows are added to, as for two CTAs on an SM: 33 K of them and a gradient all-reduce's 26 K go side by side.)
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, ACCUM ? 2 : 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
                 OutT* __restrict__ C, int M, int N, int K, long long ldc, PairPlan pl, int by_tma, int* status) {
  using Cfg = PairTile;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ __align__(8) uint64_t full_bar[6], empty_bar[6], tmem_full_bar[2], tmem_empty_bar[2];
  __shared__ uint32_t tmem_base_smem;
  __shared__ volatile int cta_abort;
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_rank());
  const int total_kb = (K + BK - 1) / BK;
  const int stages = pl.per == 2 ? 4 : 6, stage_bytes = (1 + pl.per) * Cfg::kHalfBytes;
  const int skew = min(stages, total_kb / 2);    // blocks of K by which the halves of a tile start, and end, apart
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    cta_abort = 0;
    for (int s = 0; s < 6; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tmem_full_bar[a], 1);
      mbar_init(&tmem_empty_bar[a], 8);          // the storing warps of both CTAs
    }
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    if (by_tma) tma_prefetch_desc(&tmC);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "r"(Cfg::kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                // barriers of both CTAs are there before either is used
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    // (The whole warp walks the loops of warps 0 and 1 and one thread issues: what a loop computes is then the same for all lanes, as the
    // copies and MMAs want it.)
    const bool lead = elect_one();
    RingCursor at(stages);
    const int b_half = pl.n / 2;
    const uint32_t b_bytes = B_MN ? (b_half + 63) / 64 * 8192 : b_half * 128;
    bool ok = true;
    for (int t = first; ok && t < pl.items; t += step) {
      const PairItem it = pair_item(pl, t, N);
      const int m0 = it.m0 + rank * 128, n0 = it.c0 + rank * b_half;
      for (int kb = 0; it.halves > 0 && kb < total_kb; ++kb) {
        ok = mbar_wait_warp(&empty_bar[at.stage], at.phase ^ 1u, &cta_abort, status);
        if (!ok) break;
        uint8_t* sA = smem + at.stage * stage_bytes;
        if (lead) {
          if (rank == 0) mbar_expect_tx(&full_bar[at.stage], 2 * (Cfg::kHalfBytes + it.halves * b_bytes));
          const uint32_t bar = in_first_cta(&full_bar[at.stage]);
          if (!A_MN) {
            tma_load_2d_pair(sA, &tmA, bar, kb * BK, m0);
          } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) tma_load_2d_pair(sA + i * 8192, &tmA, bar, m0 + i * 64, kb * BK);
          }
          for (int half = 0; half < it.halves; ++half) {
            uint8_t* sB = sA + (1 + half) * Cfg::kHalfBytes;
            if (!B_MN) {
              tma_load_2d_pair(sB, &tmB, bar, kb * BK, n0 + half * pl.n);
            } else {
              for (int i = 0; i < b_half; i += 64) tma_load_2d_pair(sB + i * 128, &tmB, bar, n0 + half * pl.n + i, kb * BK);
            }
          }
        }
        __syncwarp();
        at.next();
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer
    if (rank == 0) {
      const uint32_t lead = elect_one() ? 1u : 0u;
      const uint32_t idesc = umma_idesc(256, pl.n, 1, 1, A_MN ? 1 : 0, B_MN ? 1 : 0), base = smem_u32(smem);
      RingCursor at(stages);
      uint32_t acc = 0, uses = 0;                // the accumulator of the next half, and how often both have been used
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t phase) {
        ok = mbar_wait_warp(bar, phase, &cta_abort, status);
        tc_fence_after();
        return ok;
      };
      auto adesc = [&](uint32_t a, int k) { return A_MN ? umma_smem_desc_sw128(a + k * 2048, 8192, 1024) : umma_smem_desc_sw128(a + k * 32, 16, 1024); };
      auto bdesc = [&](uint32_t b, int k) { return B_MN ? umma_smem_desc_sw128(b + k * 2048, 8192, 1024) : umma_smem_desc_sw128(b + k * 32, 16, 1024); };
      for (int t = first; ok && t < pl.items; t += step) {
        const PairItem it = pair_item(pl, t, N);
        if (it.halves == 0) continue;
        const uint32_t d0 = tmem_base + acc * 256, d1 = tmem_base + (acc ^ 1) * 256;
        auto one = [&](int stage, int half, int kb) {
          const uint32_t a = base + stage * stage_bytes, b = a + (1 + half) * Cfg::kHalfBytes;
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) umma_f16_pair_if(lead, half ? d1 : d0, adesc(a, k), bdesc(b, k), idesc, (kb | k) != 0 ? 1u : 0u);
        };
        if (!wait(&tmem_empty_bar[acc], (uses & 1) ^ 1u)) break;
        if (it.halves == 1) {
          for (int kb = 0; kb < total_kb; ++kb) {
            if (!wait(&full_bar[at.stage], at.phase)) break;
            one(at.stage, 0, kb);
            umma_commit_pair_if(lead, &empty_bar[at.stage]);
            at.next();
          }
          if (!ok) break;
          umma_commit_pair_if(lead, &tmem_full_bar[acc]);
          uses += acc;
          acc ^= 1;
        } else {
          // `skew` blocks of the first half, then the same blocks of the second
          RingCursor behind = at;
          for (int kb = 0; kb < skew; ++kb, at.next()) {
            if (!wait(&full_bar[at.stage], at.phase)) break;
            one(at.stage, 0, kb);
          }
          if (!ok || !wait(&tmem_empty_bar[acc ^ 1], ((uses + acc) & 1) ^ 1u)) break;
          for (int kb = 0; kb < skew; ++kb, behind.next()) {
            one(behind.stage, 1, kb);
            umma_commit_pair_if(lead, &empty_bar[behind.stage]);
          }
          for (int kb = skew; kb < total_kb - skew; ++kb, at.next()) {
            if (!wait(&full_bar[at.stage], at.phase)) break;
            const uint32_t a = base + at.stage * stage_bytes, b0 = a + Cfg::kHalfBytes, b1 = b0 + Cfg::kHalfBytes;
#pragma unroll
            for (int k = 0; k < BK / 16; ++k)
              umma_f16_pair_twice_if(lead, d0, d1, adesc(a, k), bdesc(b0, k), bdesc(b1, k), idesc, (kb | k) != 0 ? 1u : 0u);
            umma_commit_pair_if(lead, &empty_bar[at.stage]);
          }
          if (!ok) break;
          behind = at;
          for (int kb = total_kb - skew; kb < total_kb; ++kb, at.next()) {
            if (!wait(&full_bar[at.stage], at.phase)) break;
            one(at.stage, 0, kb);
          }
          if (!ok) break;
          umma_commit_pair_if(lead, &tmem_full_bar[acc]);
          for (int kb = total_kb - skew; kb < total_kb; ++kb, behind.next()) {
            one(behind.stage, 1, kb);
            umma_commit_pair_if(lead, &empty_bar[behind.stage]);
          }
          umma_commit_pair_if(lead, &tmem_full_bar[acc ^ 1]);
          uses += 1;
        }
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5)
    const int q = warp & 3;  // TMEM lane quadrant this warp may read
    constexpr int kCols = 128 / sizeof(OutT);
    const bool vec_ok = (ldc % (16 / sizeof(OutT)) == 0) && ((reinterpret_cast<uintptr_t>(C) & 15) == 0);
    uint8_t* out = smem + Cfg::kRingBytes + q * Cfg::kOutBufs * Cfg::kOutBytes;
    int buf = 0;
    uint32_t acc = 0, uses = 0;
    bool ok = true;
    for (int t = first; ok && t < pl.items; t += step) {
      const PairItem it = pair_item(pl, t, N);
      const int row0 = it.m0 + rank * 128 + q * 32, row = row0 + lane;
      for (int half = 0; half < it.halves; ++half) {
        const int col0 = it.c0 + half * pl.n, cols = min(pl.n, N - col0);
        OutT* crow = C + static_cast<long long>(row) * ldc;
        // What is added to comes while the products are formed, two pieces of 64 columns ahead (N is a multiple of 8 here). All four would
        // take 64 registers more and the room of a gradient all-reduce's CTA beside this one.
        uint4 old[2][ACCUM && sizeof(OutT) == 2 ? 8 : 1];
        auto fetch = [&](int c) {
          if constexpr (ACCUM && sizeof(OutT) == 2) {
            if (by_tma && row < M) {
#pragma unroll
              for (int v = 0; v < 8; ++v)
                if (c * 64 + v * 8 < cols) old[c & 1][v] = *reinterpret_cast<const uint4*>(crow + col0 + c * 64 + v * 8);
            }
          }
        };
        fetch(0);
        fetch(1);
        ok = mbar_wait_warp(&tmem_full_bar[acc], uses & 1, &cta_abort, status);
        if (!ok) break;
        tc_fence_after();
        const uint32_t addr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * 256;
        if (by_tma) {
#pragma unroll
          for (int c = 0; c < 256 / kCols; ++c) {
            if (c * kCols < cols) {
              uint32_t r[kCols];
#pragma unroll
              for (int i = 0; i < kCols; i += 32) tmem_ld_32x32(addr + c * kCols + i, *reinterpret_cast<uint32_t(*)[32]>(&r[i]));
              tmem_ld_wait();
              if (lane == 0) tma_store_wait_read<Cfg::kOutBufs - 1>();       // the store that last read this buffer
              __syncwarp();
              uint8_t* piece = out + buf * Cfg::kOutBytes;
#pragma unroll
              for (int v = 0; v < 8; ++v) {
                uint4 o;
                if constexpr (sizeof(OutT) == 2) {
                  float f[8];
#pragma unroll
                  for (int j = 0; j < 8; ++j) f[j] = __uint_as_float(r[v * 8 + j]);
                  if constexpr (ACCUM) {
                    const __nv_bfloat162* o2 = reinterpret_cast<const __nv_bfloat162*>(&old[c & 1][v]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                      const float2 of = __bfloat1622float2(o2[j]);
                      f[2 * j] += of.x;
                      f[2 * j + 1] += of.y;
                    }
                  }
                  o = make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
                } else {
                  o = make_uint4(r[v * 4], r[v * 4 + 1], r[v * 4 + 2], r[v * 4 + 3]);
                }
                *reinterpret_cast<uint4*>(piece + lane * 128 + ((v ^ (lane & 7)) << 4)) = o;
              }
              if (c < 2) fetch(c + 2);
              fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                if (row0 < M) tma_store_2d(&tmC, piece, col0 + c * kCols, row0);
                tma_store_commit();
              }
              buf ^= 1;
            }
          }
        } else {
#pragma unroll 1
          for (int c = 0; c < pl.n / 32; ++c) {
            uint32_t r[32];
            tmem_ld_32x32(addr + c * 32, r);
            tmem_ld_wait();
            if (row < M && c * 32 < cols) store_columns<OutT, ACCUM>(crow, col0 + c * 32, N, vec_ok, r, false, false);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(in_first_cta(&tmem_empty_bar[acc]));
        uses += acc;
        acc ^= 1;
      }
    }
    if (lane == 0) tma_store_wait_all<0>();
  }

  // ------------------------------------------------------------ tear-down
  tc_fence_before();
  __syncthreads();
  if (cta_abort && warp == 1)   // copies and MMAs that are still in flight get a bounded moment to land before TMEM goes away
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
  __syncwarp();
  cluster_sync();               // neither CTA's shared memory goes away while the other may still reach it
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(Cfg::kTmemCols) : "memory");
  }
}

// ---------------------------------------------------------------- tensor-map cache
struct TmapKey {
  const void* p;
  uint64_t rows, cols, stride;
  uint32_t br, bc, elem;
  bool operator==(const TmapKey& o) const {
    return p == o.p && rows == o.rows && cols == o.cols && stride == o.stride && br == o.br && bc == o.bc && elem == o.elem;
  }
};
struct TmapKeyHash {
  size_t operator()(const TmapKey& k) const {
    size_t h = reinterpret_cast<size_t>(k.p) * 0x9E3779B97F4A7C15ull;
    h ^= k.rows * 0xC2B2AE3D27D4EB4Full + (h << 6) + (h >> 2);
    h ^= k.cols * 0x165667B19E3779F9ull + (h << 6) + (h >> 2);
    h ^= k.stride + (h << 6) + (h >> 2);
    h ^= (static_cast<size_t>(k.br) << 32 | k.bc << 4 | k.elem) + (h << 6) + (h >> 2);
    return h;
  }
};
std::unordered_map<TmapKey, CUtensorMap, TmapKeyHash> g_tmaps;
std::mutex g_tmap_mu;

bool cached_tmap_2d(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t stride_bytes,
                    uint32_t box_rows, uint32_t box_cols, int elem_bytes = 2) {
  TmapKey key{base, rows, cols, stride_bytes, box_rows, box_cols, static_cast<uint32_t>(elem_bytes)};
  std::lock_guard<std::mutex> lk(g_tmap_mu);
  auto it = g_tmaps.find(key);
  if (it != g_tmaps.end()) {
    *out = it->second;
    return true;
  }
  if (!make_tmap_2d(out, base, elem_bytes, rows, cols, stride_bytes, box_rows, box_cols, true)) return false;
  if (g_tmaps.size() > 8192) g_tmaps.clear();
  g_tmaps.emplace(key, *out);
  return true;
}

template <int BN, bool A_MN, bool B_MN, typename OutT, bool ACCUM>
int launch_cfg(const CUtensorMap& ta, const CUtensorMap& tb, void* C, int M, int N, int K, long long ldc, int max_ctas,
               cudaStream_t stream, int split_k = 1, GroupArgs grp = GroupArgs{nullptr, 0, 0, 0, 0}) {
  using Cfg = GemmCfg<BN>;
  auto kern = gemm_bf16_kernel<BN, A_MN, B_MN, OutT, ACCUM>;
  static PerDeviceFlag attr_set;
  if (attr_set.unset()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set.set();
  }
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN) * ((grp.offsets && grp.mode == 2) ? grp.groups : split_k);
  int grid = sm_count();
  if (max_ctas > 0 && max_ctas < grid) grid = max_ctas;
  if (tiles < grid) grid = tiles;
  kern<<<grid, kGemmThreads, Cfg::kSmemBytes, stream>>>(ta, tb, static_cast<OutT*>(C), M, N, K, ldc,
                                                        device_status_word(), split_k, grp);
  return static_cast<int>(cudaGetLastError());
}

template <int BN, bool A_MN, bool B_MN>
int launch_out(const CUtensorMap& ta, const CUtensorMap& tb, void* C, int M, int N, int K, long long ldc, int out_f32,
               int accumulate, int max_ctas, cudaStream_t s) {
  if (out_f32) {
    return accumulate ? launch_cfg<BN, A_MN, B_MN, float, true>(ta, tb, C, M, N, K, ldc, max_ctas, s)
                      : launch_cfg<BN, A_MN, B_MN, float, false>(ta, tb, C, M, N, K, ldc, max_ctas, s);
  }
  return accumulate ? launch_cfg<BN, A_MN, B_MN, __nv_bfloat16, true>(ta, tb, C, M, N, K, ldc, max_ctas, s)
                    : launch_cfg<BN, A_MN, B_MN, __nv_bfloat16, false>(ta, tb, C, M, N, K, ldc, max_ctas, s);
}

template <int BN>
int launch_major(const CUtensorMap& ta, const CUtensorMap& tb, void* C, int M, int N, int K, long long ldc, int a_mn,
                 int b_mn, int out_f32, int accumulate, int max_ctas, cudaStream_t s) {
  if (!a_mn && !b_mn) return launch_out<BN, false, false>(ta, tb, C, M, N, K, ldc, out_f32, accumulate, max_ctas, s);
  if (!a_mn && b_mn) return launch_out<BN, false, true>(ta, tb, C, M, N, K, ldc, out_f32, accumulate, max_ctas, s);
  if (a_mn && !b_mn) return launch_out<BN, true, false>(ta, tb, C, M, N, K, ldc, out_f32, accumulate, max_ctas, s);
  return launch_out<BN, true, true>(ta, tb, C, M, N, K, ldc, out_f32, accumulate, max_ctas, s);
}

template <bool A_MN, bool B_MN, typename OutT, bool ACCUM>
int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, void* C, int M, int N, int K, long long ldc, const PairPlan& plan, cudaStream_t stream) {
  auto kern = gemm_pair_kernel<A_MN, B_MN, OutT, ACCUM>;
  static PerDeviceFlag attr_set;
  if (attr_set.unset()) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairTile::kSmemBytes);
    if (e != cudaSuccess) return static_cast<int>(e);
    attr_set.set();
  }
  // Stores by TMA want rows that start on 16 bytes. Added to (ACCUM), bf16 rows are also read 16 bytes at a time up to N, and fp32 rows,
  // of which a thread cannot hold enough ahead, go the plain way.
  CUtensorMap tc{};
  const int by_tma = (reinterpret_cast<uintptr_t>(C) & 15) == 0 && ldc * sizeof(OutT) % 16 == 0 && (!ACCUM || (sizeof(OutT) == 2 && N % 8 == 0));
  if (by_tma && !cached_tmap_2d(&tc, C, M, N, ldc * sizeof(OutT), 32, 128 / sizeof(OutT), sizeof(OutT))) return -3;
  const int pairs = sm_count() / 2;
  kern<<<2 * (plan.items < pairs ? plan.items : pairs), kGemmThreads, PairTile::kSmemBytes, stream>>>(
      ta, tb, tc, static_cast<OutT*>(C), M, N, K, ldc, plan, by_tma, device_status_word());
  return static_cast<int>(cudaGetLastError());
}

template <bool A_MN, bool B_MN>
int launch_pair_out(const CUtensorMap& ta, const CUtensorMap& tb, void* C, int M, int N, int K, long long ldc, int out_f32, int accumulate,
                    const PairPlan& pl, cudaStream_t s) {
  if (out_f32)
    return accumulate ? launch_pair<A_MN, B_MN, float, true>(ta, tb, C, M, N, K, ldc, pl, s)
                      : launch_pair<A_MN, B_MN, float, false>(ta, tb, C, M, N, K, ldc, pl, s);
  return accumulate ? launch_pair<A_MN, B_MN, __nv_bfloat16, true>(ta, tb, C, M, N, K, ldc, pl, s)
                    : launch_pair<A_MN, B_MN, __nv_bfloat16, false>(ta, tb, C, M, N, K, ldc, pl, s);
}

PairPlan make_pair_plan(int M, int N, int n, int per) {
  const int num_m = (M + 255) / 256, num_w = (N + per * n - 1) / (per * n);
  const int tiles = num_m * num_w, pairs = sm_count() / 2, rest = tiles % pairs;
  const int full = per == 2 && 2 * rest <= pairs ? tiles - rest : tiles;
  // rows of tiles that are worked on together: with few columns of tiles a round covers all of them (17000 x 4096 x 14336: 8 1473, 16 1485 us),
  // with many, more rows keep what it reads small (8192 x 28672 x 4096: 16 1412, 8 1435)
  return {n, per, num_w >= 16 ? 16 : 8, num_m, num_w, full, full + 2 * (tiles - full)};
}

// What a product takes with tiles of a kind, up to a factor that they share: the tiles that one SM (or pair) works on in turn, times the
// columns of a tile, times how much slower a column is than in the widest ones. The factors are fitted to the times of all kinds at 351 products of training
// and prompts (forward and both gradients; 136 - 17000 rows, 256 - 32000 columns, depths 136 - 32000): what is chosen takes 2.4 % more than the best kind in
// the mean, nothing in the median, at most 27 % (launches of 7 us, and gradients of 512 - 1024 rows; `kernel_cases.py --case gemm_kinds` has the
// forward ones). Deep products want whole tiles of 256 x 512 (input gradient 4096 x 4096 x 28672: 744 us against 759 for halves by themselves), others halves,
// whose stores start earlier (all in turn, 60 ms at a time: weight gradients 128256 x 4096 x 4096 2878 against 3792, 4096 x 14336 x 4096 339 against 422,
// forward 8192 x 28672 x 4096 1291 against 1424). Widths of 192 fit where 256 would leave most of a round empty (3003 x 2048 x 8192: 72 against 93), but a
// column of theirs costs more, of whole tiles too (8192 x 6144 x 4096: 327 against 301 for halves of 256; input gradient 1024 x 14336 x 4096
// 115 against 106). Tiles of one SM remain for up to 128 rows, for few tiles
// (296 x 2176 x 5120: 64 columns 18.5, pairs 23.8 at best) and where the last pair of row tiles would be half empty (528 x 44384 x 3264: 142 against 166).
double pair_cost(const PairPlan& pl, int K) {
  const int pairs = sm_count() / 2, halves = pl.items - pl.full;
  const int rounds = (pl.full + pairs - 1) / pairs * pl.per + (halves > 0 ? 1 : 0);
  const double slow = (pl.per == 2 ? 1.0 : K >= 6144 ? 1.05 : K >= 3072 ? 0.98 : 0.95) *
                      (pl.n == 256 ? 1.0 : pl.n == 128 ? 1.25 : 1.08);
  return rounds * pl.n * slow;
}
double cta_cost(int M, int N, int K, int bn) {
  const long long tiles = static_cast<long long>((M + BM - 1) / BM) * ((N + bn - 1) / bn);
  return static_cast<double>((tiles + sm_count() - 1) / sm_count()) * bn * (bn == 256 ? (K >= 3072 ? 1.06 : 1.15) : bn == 128 ? 1.33 : bn == 64 ? 2.25 : 4.0);
}

// Columns of the tiles of one SM, or (pair) the cut for pairs of SMs.
struct Tiles {
  int bn;
  bool pair;
  PairPlan plan;
};
Tiles choose_tiles(int M, int N, int K, int max_ctas) {
  Tiles t{};
  const int sms = sm_count();
  const long long mt = (M + BM - 1) / BM;
  auto tiles = [&](int b) { return mt * ((N + b - 1) / b); };
  // largest tile that still gives every SM work; decode-shaped calls (few rows) stream the weight matrix
  // and want as many CTAs pulling on HBM as possible, so they go down to 32-column tiles
  if (N >= 256 && tiles(256) >= sms) t.bn = 256;
  else if (N >= 128 && tiles(128) >= sms) t.bn = 128;
  else if (N >= 64 && tiles(64) >= sms) t.bn = 64;
  else if (N >= 128 && tiles(128) * 2 >= sms && mt > 2) t.bn = 128;
  else t.bn = (N >= 64 && tiles(32) > 2 * sms) ? 64 : 32;
  // More than one tile of rows, and columns for a wide one: the cheapest kind.
  if (max_ctas <= 0 && M > 128 && N >= 192) {
    double best = cta_cost(M, N, K, t.bn);
    for (const int b : {64, 128, 256})
      if (const double cost = cta_cost(M, N, K, b); cost < best) {
        best = cost;
        t.bn = b;
      }
    constexpr int kinds[][2] = {{256, 2}, {256, 1}, {192, 2}, {192, 1}, {128, 1}};
    for (const auto& kind : kinds) {
      const PairPlan pl = make_pair_plan(M, N, kind[0], kind[1]);
      if (const double cost = pair_cost(pl, K); cost < best) {
        best = cost;
        t.plan = pl;
        t.pair = true;
      }
    }
  }
  return t;
}

int run_gemm(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int a_mn, int b_mn, int out_f32,
             int accumulate, const Tiles& t, int max_ctas, cudaStream_t s) {
  CUtensorMap ta, tb;
  bool ok;
  if (!a_mn) ok = cached_tmap_2d(&ta, A, M, K, lda * 2, BM, BK);
  else ok = cached_tmap_2d(&ta, A, K, M, lda * 2, BK, 64);
  if (!ok) return -3;
  if (!b_mn) ok = cached_tmap_2d(&tb, B, N, K, ldb * 2, t.pair ? t.plan.n / 2 : t.bn, BK);
  else ok = cached_tmap_2d(&tb, B, K, N, ldb * 2, BK, 64);
  if (!ok) return -3;
  if (t.pair) {
    if (!a_mn)
      return b_mn ? launch_pair_out<false, true>(ta, tb, C, M, N, K, ldc, out_f32, accumulate, t.plan, s)
                  : launch_pair_out<false, false>(ta, tb, C, M, N, K, ldc, out_f32, accumulate, t.plan, s);
    return b_mn ? launch_pair_out<true, true>(ta, tb, C, M, N, K, ldc, out_f32, accumulate, t.plan, s)
                : launch_pair_out<true, false>(ta, tb, C, M, N, K, ldc, out_f32, accumulate, t.plan, s);
  }
  switch (t.bn) {
    case 256: return launch_major<256>(ta, tb, C, M, N, K, ldc, a_mn, b_mn, out_f32, accumulate, max_ctas, s);
    case 128: return launch_major<128>(ta, tb, C, M, N, K, ldc, a_mn, b_mn, out_f32, accumulate, max_ctas, s);
    case 64: return launch_major<64>(ta, tb, C, M, N, K, ldc, a_mn, b_mn, out_f32, accumulate, max_ctas, s);
    default: return launch_major<32>(ta, tb, C, M, N, K, ldc, a_mn, b_mn, out_f32, accumulate, max_ctas, s);
  }
}

bool gemm_operands_ok(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb) {
  return M > 0 && N > 0 && K > 0 && !(reinterpret_cast<uintptr_t>(A) & 15) && !(reinterpret_cast<uintptr_t>(B) & 15) && lda % 8 == 0 && ldb % 8 == 0;
}

}  // namespace
}  // namespace tsb

// C[M,N] (+)= op(A) * op(B) with bf16 inputs and fp32 accumulation.
//   a_mn == 0: A is row-major [M, K] (row stride lda elements);  a_mn == 1: A is row-major [K, M].
//   b_mn == 0: B is row-major [N, K] (row stride ldb elements);  b_mn == 1: B is row-major [K, N].
//   C is row-major [M, N] with row stride ldc; bf16, or fp32 when out_f32 != 0; accumulate != 0 adds
//   into the existing contents of C.
// Requirements: A and B 16-byte aligned with row strides that are multiples of 8 elements.
// block_n: 0 = choose, else 32 / 64 / 128 / 256. max_ctas: 0 = one CTA per SM, else a cap (used when some SMs are
// reserved for a concurrent communication kernel).
// Returns 0, a cudaError_t, or -2 (bad argument) / -3 (tensor map encoding failed).
TSB_EXPORT int tsb_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda,
                             long long ldb, long long ldc, int a_mn, int b_mn, int out_f32, int accumulate,
                             int block_n, int max_ctas, void* stream) {
  using namespace tsb;
  if (!gemm_operands_ok(A, B, M, N, K, lda, ldb)) return -2;
  Tiles t = block_n == 0 ? choose_tiles(M, N, K, max_ctas) : Tiles{block_n, false, {}};
  if (t.bn == 32 && b_mn) t.bn = 64;  // an N-major B tile is built from 64-column (128-byte) boxes
  if (t.bn != 32 && t.bn != 64 && t.bn != 128 && t.bn != 256) return -2;
  return run_gemm(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_f32, accumulate, t, max_ctas, static_cast<cudaStream_t>(stream));
}

// How tsb_gemm_bf16 (block_n = 0, max_ctas = 0) cuts a product, host array of four: columns of a tile; 1 or 2 of them per tile of a pair of SMs, 0 where
// the tiles are one SM's; whole tiles; items (whole tiles, and two halves for each of the others).
TSB_EXPORT int tsb_gemm_bf16_plan(int M, int N, int K, int* out) {
  using namespace tsb;
  if (M <= 0 || N <= 0 || K <= 0) return -2;
  const Tiles t = choose_tiles(M, N, K, 0);
  out[0] = t.pair ? t.plan.n : t.bn;
  out[1] = t.pair ? t.plan.per : 0;
  out[2] = t.plan.full;
  out[3] = t.plan.items;
  return 0;
}

// tsb_gemm_bf16 with the kind of tiles given for pairs of SMs, to compare what choose_tiles chooses from: n = 256 or 192 with per = 1 or 2, or 128
// with 1. More than 128 rows, 192 columns at least.
TSB_EXPORT int tsb_gemm_bf16_pairs(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb, long long ldc, int a_mn,
                                   int b_mn, int out_f32, int accumulate, int n, int per, void* stream) {
  using namespace tsb;
  if (!gemm_operands_ok(A, B, M, N, K, lda, ldb) || M <= 128 || N < 192) return -2;
  if (!((n == 256 || n == 192) && (per == 1 || per == 2)) && !(n == 128 && per == 1)) return -2;
  const Tiles t{0, true, make_pair_plan(M, N, n, per)};
  return run_gemm(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_f32, accumulate, t, 0, static_cast<cudaStream_t>(stream));
}

// Grouped GEMM for mixture-of-experts layers; `offsets` (int32 [groups + 1], multiples of 128) stays on the device.
//   mode 1 (rows grouped):  C[r, :] = A[r, :] * op(B[g(r)])  for the row blocks below offsets[groups].
//       A [rows_cap, K] bf16 (lda), C [rows_cap, N] bf16 (ldc); rows_cap >= offsets[groups] is the allocated height.
//       b_mn = 0: B[g] is [N, K];  b_mn = 1: B[g] is [K, N]  (row stride ldb); B[g] starts b_group_stride elements
//       after B[g - 1] (a multiple of ldb: the groups need not be packed, e.g. expert weights in a flat arena). act = 1: relu(C)^2.
//   mode 2 (reduction grouped, expert weight gradient):  C[g] (+)= A[rows of g, :]^T * B[rows of g, :]
//       A [rows_cap, M] bf16 (lda), B [rows_cap, N] bf16 (ldb), C[g] [M, N] fp32 or bf16 (ldc), C[g] starting
//       c_group_stride elements after C[g - 1].
// Returns 0, a cudaError_t, -2 (bad argument) or -3 (tensor map encoding failed).
TSB_EXPORT int tsb_gemm_grouped(const void* A, const void* B, void* C, const int* offsets, int groups, int mode,
                                int rows_cap, int M, int N, int K, long long lda, long long ldb, long long ldc, int b_mn,
                                long long b_group_stride, long long c_group_stride, int out_f32, int accumulate, int act,
                                void* stream) {
  using namespace tsb;
  if (act < 0 || act > 1 || (act && mode != 1)) return -2;
  if (!offsets || groups < 1 || groups > 1024 || rows_cap <= 0 || rows_cap % BM || N <= 0) return -2;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda % 8) || (ldb % 8)) return -2;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  CUtensorMap ta, tb;
  if (mode == 1) {
    if (K <= 0 || K % 8 || out_f32 || accumulate) return -2;
    if (b_mn && (K % BK)) return -2;  // the stacked [groups * K, N] map must not read across a group boundary
    const int bn = (N >= 256) ? 256 : (N >= 128 ? 128 : 64);
    if (!cached_tmap_2d(&ta, A, rows_cap, K, lda * 2, BM, BK)) return -3;
    if (b_group_stride <= 0 || b_group_stride % ldb) return -2;
    const long long grows = b_group_stride / ldb;  // rows of the stacked map per group
    if (grows < (b_mn ? K : N)) return -2;
    const uint64_t map_rows = static_cast<uint64_t>(groups - 1) * grows + (b_mn ? K : N);
    const bool ok = b_mn ? cached_tmap_2d(&tb, B, map_rows, N, ldb * 2, BK, 64)
                         : cached_tmap_2d(&tb, B, map_rows, K, ldb * 2, bn, BK);
    if (!ok) return -3;
    GroupArgs g{offsets, groups, 1, grows, 0};
    g.act = act;
    auto go = [&](auto bn_tag, auto bmn_tag) {
      return launch_cfg<decltype(bn_tag)::value, false, decltype(bmn_tag)::value, __nv_bfloat16, false>(
          ta, tb, C, rows_cap, N, K, ldc, 0, s, 1, g);
    };
    using T = std::true_type;
    using F = std::false_type;
    if (bn == 256) return b_mn ? go(std::integral_constant<int, 256>{}, T{}) : go(std::integral_constant<int, 256>{}, F{});
    if (bn == 128) return b_mn ? go(std::integral_constant<int, 128>{}, T{}) : go(std::integral_constant<int, 128>{}, F{});
    return b_mn ? go(std::integral_constant<int, 64>{}, T{}) : go(std::integral_constant<int, 64>{}, F{});
  }
  if (mode == 2) {
    if (M <= 0 || M % 8 || N % 8) return -2;
    const int bn = (N >= 256) ? 256 : (N >= 128 ? 128 : 64);
    if (!cached_tmap_2d(&ta, A, rows_cap, M, lda * 2, BK, 64)) return -3;
    if (!cached_tmap_2d(&tb, B, rows_cap, N, ldb * 2, BK, 64)) return -3;
    if (c_group_stride < static_cast<long long>(M - 1) * ldc + N) return -2;
    GroupArgs g{offsets, groups, 2, 0, c_group_stride};
    auto go = [&](auto bn_tag) {
      constexpr int kBn = decltype(bn_tag)::value;
      if (out_f32)
        return accumulate ? launch_cfg<kBn, true, true, float, true>(ta, tb, C, M, N, rows_cap, ldc, 0, s, 1, g)
                          : launch_cfg<kBn, true, true, float, false>(ta, tb, C, M, N, rows_cap, ldc, 0, s, 1, g);
      return accumulate ? launch_cfg<kBn, true, true, __nv_bfloat16, true>(ta, tb, C, M, N, rows_cap, ldc, 0, s, 1, g)
                        : launch_cfg<kBn, true, true, __nv_bfloat16, false>(ta, tb, C, M, N, rows_cap, ldc, 0, s, 1, g);
    };
    if (bn == 256) return go(std::integral_constant<int, 256>{});
    if (bn == 128) return go(std::integral_constant<int, 128>{});
    return go(std::integral_constant<int, 64>{});
  }
  return -2;
}

// Row-grouped GEMM (mode 1 above) whose result rows are scattered to peer-mapped buffers instead of a local C:
// row r goes to peer_out[tags[r] >> 24] + (tags[r] & 0xFFFFFF) * ld_out when tags[r] >= 0 (and the slot is below
// peer_rows), nowhere otherwise. peer_out: `world` (<= 8) device pointers as mapped in this process, 16-byte aligned,
// ld_out % 8 == 0. Plain stores: the caller orders them with its own barrier (e.g. tsb_symm_barrier).
TSB_EXPORT int tsb_gemm_grouped_scatter(const void* A, const void* B, const int* offsets, int groups, int rows_cap, int N,
                                        int K, long long lda, long long ldb, int b_mn, long long b_group_stride,
                                        const int* tags, void* const* peer_out, int world, long long peer_rows,
                                        long long ld_out, void* stream) {
  using namespace tsb;
  if (!offsets || !tags || !peer_out || world < 1 || world > 8 || groups < 1 || groups > 1024 || rows_cap <= 0 ||
      rows_cap % BM || N <= 0 || K <= 0 || K % 8 || ld_out % 8 || peer_rows <= 0 || peer_rows > 0xFFFFFF)
    return -2;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda % 8) || (ldb % 8)) return -2;
  if (b_mn && (K % BK)) return -2;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  CUtensorMap ta, tb;
  const int bn = (N >= 256) ? 256 : (N >= 128 ? 128 : 64);
  if (!cached_tmap_2d(&ta, A, rows_cap, K, lda * 2, BM, BK)) return -3;
  if (b_group_stride <= 0 || b_group_stride % ldb) return -2;
  const long long grows = b_group_stride / ldb;
  if (grows < (b_mn ? K : N)) return -2;
  const uint64_t map_rows = static_cast<uint64_t>(groups - 1) * grows + (b_mn ? K : N);
  const bool ok = b_mn ? cached_tmap_2d(&tb, B, map_rows, N, ldb * 2, BK, 64)
                       : cached_tmap_2d(&tb, B, map_rows, K, ldb * 2, bn, BK);
  if (!ok) return -3;
  GroupArgs g{offsets, groups, 1, grows, 0};
  g.row_tags = tags;
  g.peer_rows = peer_rows;
  for (int r = 0; r < world; ++r) {
    if (!peer_out[r] || (reinterpret_cast<uintptr_t>(peer_out[r]) & 15)) return -2;
    g.peer_out[r] = peer_out[r];
  }
  void* C = peer_out[0];   // only its alignment is looked at
  auto go = [&](auto bn_tag, auto bmn_tag) {
    return launch_cfg<decltype(bn_tag)::value, false, decltype(bmn_tag)::value, __nv_bfloat16, false>(
        ta, tb, C, rows_cap, N, K, ld_out, 0, s, 1, g);
  };
  using T = std::true_type;
  using F = std::false_type;
  if (bn == 256) return b_mn ? go(std::integral_constant<int, 256>{}, T{}) : go(std::integral_constant<int, 256>{}, F{});
  if (bn == 128) return b_mn ? go(std::integral_constant<int, 128>{}, T{}) : go(std::integral_constant<int, 128>{}, F{});
  return b_mn ? go(std::integral_constant<int, 64>{}, T{}) : go(std::integral_constant<int, 64>{}, F{});
}

// Split-K variant for decode-shaped calls (few rows, the weight matrix is streamed once): the K range is cut into
// `split_k` slices that run as independent work items, so that all SMs pull on HBM, and their fp32 partial sums are
// added into C32 with vector atomics. C32 (fp32 [M, N], row stride ldc) must be zero on entry. A is [M, K] row-major,
// B is [N, K] (b_mn = 0) or [K, N] (b_mn = 1). block_n: 64 or 128.
TSB_EXPORT int tsb_gemm_bf16_splitk(const void* A, const void* B, float* C32, int M, int N, int K, long long lda,
                                    long long ldb, long long ldc, int b_mn, int split_k, int block_n, void* stream) {
  using namespace tsb;
  if (M <= 0 || N <= 0 || K <= 0 || split_k < 1 || split_k > 64) return -2;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda % 8) || (ldb % 8) || (ldc % 4))
    return -2;
  const int bn = block_n == 64 ? 64 : 128;
  CUtensorMap ta, tb;
  if (!cached_tmap_2d(&ta, A, M, K, lda * 2, BM, BK)) return -3;
  if (!(b_mn ? cached_tmap_2d(&tb, B, K, N, ldb * 2, BK, 64) : cached_tmap_2d(&tb, B, N, K, ldb * 2, bn, BK))) return -3;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (bn == 128)
    return b_mn ? launch_cfg<128, false, true, float, false>(ta, tb, C32, M, N, K, ldc, 0, s, split_k)
                : launch_cfg<128, false, false, float, false>(ta, tb, C32, M, N, K, ldc, 0, s, split_k);
  return b_mn ? launch_cfg<64, false, true, float, false>(ta, tb, C32, M, N, K, ldc, 0, s, split_k)
              : launch_cfg<64, false, false, float, false>(ta, tb, C32, M, N, K, ldc, 0, s, split_k);
}

// C[M, N] (bf16) whose column ranges read different inputs: columns [starts[i], starts[i + 1]) are A_i[M, K] * B[N, K]^T, A_i starting
// i * a_rows rows after A (a_rows >= M). Host array `starts` ascends from 0 in multiples of 128; n <= 8. Alignment as tsb_gemm_bf16.
TSB_EXPORT int tsb_gemm_bf16_inputs(const int* starts, const void* A, const void* B, void* C, int n, int M, int N, int K, long long a_rows,
                                    long long lda, long long ldb, long long ldc, void* stream) {
  using namespace tsb;
  if (n < 1 || n > 8 || M <= 0 || N <= 0 || K <= 0 || a_rows < M || starts[0] != 0) return -2;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) || (lda % 8) || (ldb % 8)) return -2;
  GroupArgs g{nullptr, 0, 0, 0, 0};
  g.inputs = n;
  g.a_group_rows = static_cast<int>(a_rows);
  bool wide = true;
  for (int i = 0; i < n; ++i) {
    if (starts[i] % 128 || (i && starts[i] <= starts[i - 1]) || starts[i] >= N) return -2;
    g.col_start[i] = starts[i];
    wide = wide && starts[i] % 256 == 0;
  }
  const long long mt = (M + BM - 1) / BM;
  const int bn = wide && mt * ((N + 255) / 256) >= sm_count() ? 256 : mt * ((N + 127) / 128) >= sm_count() ? 128 : 64;
  CUtensorMap ta, tb;
  if (!cached_tmap_2d(&ta, A, (n - 1) * a_rows + M, K, lda * 2, BM, BK) || !cached_tmap_2d(&tb, B, N, K, ldb * 2, bn, BK)) return -3;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (bn == 256) return launch_cfg<256, false, false, __nv_bfloat16, false>(ta, tb, C, M, N, K, ldc, 0, s, 1, g);
  if (bn == 128) return launch_cfg<128, false, false, __nv_bfloat16, false>(ta, tb, C, M, N, K, ldc, 0, s, 1, g);
  return launch_cfg<64, false, false, __nv_bfloat16, false>(ta, tb, C, M, N, K, ldc, 0, s, 1, g);
}
