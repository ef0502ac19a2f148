// FlashAttention backward on tcgen05 tensor cores (bf16, head_dim 64 or 128, causal or full, GQA).
//
// The reference has no attention backward kernel: it differentiates the matmul -> softmax -> matmul
// composite and keeps the [B, H, S, S] probabilities (src/ops/cpu/Attention.cpp:232-242,272-303). This
// kernel recomputes P from the saved log-sum-exp and never materialises an S x S tensor.
//
// One CTA per (128-key tile, KV head, batch). It keeps K_j and V_j in shared memory and the dK_j / dV_j
// accumulators in TMEM (fp32) while it walks over every query tile that can see the key tile, for each of
// the H / Hkv query heads that share the KV head (so the GQA reduction costs nothing). Scores are formed with keys
// as rows, so that P^T and dS^T are what dV and dK need as they come out. Per step:
//   S^T = K_j Q_i^T, dP^T = V_j dO_i^T                    (tensor core -> TMEM)
//   P^T = exp2(S^T * c - lse_i)   dS^T = P^T * (dP^T - delta_i)
//   dV_j += P^T dO_i   dK_j += dS^T Q_i                   (P^T and dS^T in TMEM, over S^T and dP^T)
//   dQ_i = dS K_j                                         (dS^T in shared memory, read M-major)
// The softmax scale is applied to dK and dQ at the end, in fp32.
//
//   warps 0-3, 4-7  P and dS of query columns 0-63 / 64-127, one key row per thread; at the end dK / dV out
//   warps 8-11      dQ_i from TMEM into an fp32 scratch that holds the four-float chunks of 32 rows side by side, so that what a
//                   warp adds is contiguous. Heads of 64: bulk reductions out of shared memory, because atomics of these warps
//                   queue up in front of the loads and stores of warps 0-7 (4 x 1500 tokens, 16 heads, full: 278 -> 258 us).
//                   Heads of 128: vector atomics, because twice the bytes meet the rate of the L2 (about 1700 bytes a clock,
//                   5500 clocks a step of all SMs), of which bulk reductions reach less (16384 tokens, 32 / 8 heads, causal: 6.4
//                   against 6.6 ms).
//   warp 12         TMA producer       warp 13   allocates TMEM, issues the MMAs      (warps 14, 15 only give their registers)
// Order of the MMAs of step i. Heads of 128, whose dQ lies over dP: dP_i, dV_i, S_{i+1}, dK_i, dQ_i. dP_i needs no probabilities and S_{i+1} no
// gradients, so that P of step i + 1 is formed while dK_i, dQ_i and dP_{i+1} run, and dS_i while dV_i and S_{i+1} do. Heads of 64, whose dQ has columns
// of its own: dV_i, S_{i+1}, dK_i, dP_{i+1}, dQ_i (dP_0 in front of all). There dP_{i+1} being ready says nothing about dQ_i, so that of dS_{i+1} in
// shared memory only the compute warps' wait for dQ_i keeps dS_i from being overwritten under it.
//
// Measured, all of the backward pass (32 / 8 heads of 128, causal), L2 flushed: 2 x 4096 tokens 0.83 ms, 16384 tokens 6.2 ms (885 TFLOP/s; 0.87
// and 6.4 with one lane's issue loops), against 1.89 and 13.6 for four warps that went through scores, P, dS and dQ of a tile one after another;
// 16 heads of 64, 4 x 1500 tokens, full: 382 -> 208 us. What bounds it now: the atomics of dQ for heads of 128 (4.6 ms without them; the stores of dS
// queue up behind them), for heads of 64 the two phases of the compute warps, P 1340 and dS 920 of 3200 clocks a step, of which the tensor core works 1280.
//
// A kernel before it writes delta_i = rowsum(dO_i * O_i) and lse_i in units of log 2 (+inf where a row sees no key or does not
// exist: P is 0 there) and zeroes the scratch; one after it turns dQ into bf16.
#include "common.cuh"

#include <type_traits>

namespace tsb {

bool make_bshd_tmap(CUtensorMap* out, const void* base, int B, int S, int Hn, int D, long long sb, long long ss,
                    long long sh, int box_rows);

namespace {

constexpr int kBwdThreads = 512;
constexpr int BT = 128;  // tile edge (queries and keys)
// Registers per thread: 128 at the launch; after it 160 for warps 0-7, 136 for 8-11, 56 for 12-15 (256 x 160 + 128 x 136 +
// 128 x 56 = 512 x 128).
constexpr int kBwdComputeRegs = 160, kBwdReduceRegs = 136, kBwdOtherRegs = 56;

template <int D>
struct BwdCfg {
  static constexpr int kHalves = D / 64;
  static constexpr int kTileBytes = 128 * D * 2;
  static constexpr int kQStages = 2, kDOStages = D == 128 ? 1 : 2;
  static constexpr int kRowBytes = 2 * BT * 4;      // lse and delta of a query tile, beside each stage of Q
  static constexpr int kPieces = D == 64 ? 3 : 0, kPieceBytes = 32 * 16 * 4;   // a warp's ring of pieces of dQ, 32 rows x 16 columns
  static constexpr int kSmemBytes =
      (2 + kQStages + kDOStages) * kTileBytes + BT * BT * 2 + kQStages * kRowBytes + 4 * kPieces * kPieceBytes + 1024;
  static constexpr bool kOwnDQ = D == 64;           // heads of 64 leave room for dQ; with 128 columns it lies over dP
  static constexpr int kColS = 0, kColDP = 128, kColDV = 256, kColDK = 256 + D, kColDQ = D == 128 ? kColDP : 384;
};

struct BwdParams {
  const float* lse2;   // [B, H, n_q * 128]: log-sum-exp * log2 e, +inf for rows without a visible key and for rows that fill up
  const float* delta;  // the same, 0 for rows that fill up
  float* dq_acc;       // [B, H, Sq, D] fp32, zero-initialised; each 32 rows (n at the end of Sq) as [D / 4][n][4]
  __nv_bfloat16* dk;
  __nv_bfloat16* dv;
  int Sq, Sk, H, Hkv, n_q;
  long long sb, ss, sh;      // of dk and dv
  float scale, scale_log2;
  int causal;
  int* status;
};

template <int ROWS>
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t base, int ks) {
  const int half = ks >> 2;
  return umma_smem_desc_sw128(base + half * (ROWS * 128) + (ks & 3) * 32, 16, 1024);
}
__device__ __forceinline__ uint64_t mnmajor_desc(uint32_t base, int ks, uint32_t half_stride) {
  return umma_smem_desc_sw128(base + ks * 2048, half_stride, 1024);
}

template <int D>
__global__ void __launch_bounds__(kBwdThreads, 1)
flash_bwd_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmDO, BwdParams p) {
  using Cfg = BwdCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + Cfg::kTileBytes;
  uint8_t* sQ = sV + Cfg::kTileBytes;
  uint8_t* sDO = sQ + Cfg::kQStages * Cfg::kTileBytes;
  uint8_t* sDS = sDO + Cfg::kDOStages * Cfg::kTileBytes;
  uint8_t* sRow = sDS + BT * BT * 2;
  uint8_t* sPiece = sRow + Cfg::kQStages * Cfg::kRowBytes;

  __shared__ __align__(8) uint64_t kv_full, q_full[2], q_empty[2], do_full[2], do_empty[2], s_full, p_full, dp_full, ds_full, dq_full, dq_read;
  __shared__ uint32_t tmem_base_smem;
  __shared__ volatile int cta_abort;

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
  const int lane = threadIdx.x & 31;
  // KV heads on the fast axis: under causal masking the first key tiles, seen by the most queries, all start first. (Both on x: key
  // tiles may be more than the other axes take.)
  const int j = blockIdx.x / p.Hkv;  // key tile
  const int hk = blockIdx.x - j * p.Hkv;
  const int b = blockIdx.z;
  const int G = p.H / p.Hkv;
  const int c0 = j * BT;
  const int offset = p.Sk - p.Sq;
  int i_min = 0;
  if (p.causal) {
    const int first = c0 - offset;  // first query row that can see key c0
    i_min = first <= 0 ? 0 : first / BT;
  }
  const int per_head = p.n_q > i_min ? p.n_q - i_min : 0;
  const int n_iter = per_head * G;
  // without a causal mask the CTAs of a head start at different query tiles: their atomics go to different tiles of dQ
  const int rot = p.causal || per_head == 0 ? 0 : j % per_head;
  // step t: query tile i of head h; next() goes on to step t + 1
  struct Walk {
    int r, i, h;
  };
  const Walk first = {0, i_min + rot, hk * G};
  auto next = [&](Walk& w) {
    ++w.i;
    if (w.i == p.n_q) w.i = i_min;
    if (++w.r == per_head) {
      w = {0, i_min + rot, w.h + 1};
    }
  };

  if (threadIdx.x == 0) {
    cta_abort = 0;
    mbar_init(&kv_full, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&q_full[i], 1);
      mbar_init(&q_empty[i], 1);
      mbar_init(&do_full[i], 1);
      mbar_init(&do_empty[i], 1);
    }
    mbar_init(&s_full, 1);
    mbar_init(&p_full, 256);
    mbar_init(&dp_full, 1);
    mbar_init(&ds_full, 256);
    mbar_init(&dq_full, 1);
    mbar_init(&dq_read, 128);
    mbar_fence_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmDO);
  }
  if (warp == 13) {
    tmem_alloc(&tmem_base_smem, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_smem;

  if (warp >= 12) {
    warpgroup_regs_dec<kBwdOtherRegs>();
    if (warp == 12) {
      // ---------------------------------------------------------------- TMA producer
      if (n_iter > 0) {
        const bool lead = elect_one();       // (the loops of warps 12 and 13 are walked by the whole warp)
        if (lead) {
          mbar_expect_tx(&kv_full, 2 * Cfg::kTileBytes);
#pragma unroll
          for (int hf = 0; hf < Cfg::kHalves; ++hf) {
            tma_load_4d(sK + hf * 16384, &tmK, &kv_full, hf * 64, c0, hk, b);
            tma_load_4d(sV + hf * 16384, &tmV, &kv_full, hf * 64, c0, hk, b);
          }
        }
        Walk w = first;
        for (int t = 0; t < n_iter; ++t, next(w)) {
          const int i = w.i, h = w.h;
          const int qs = t % Cfg::kQStages, ds = t % Cfg::kDOStages;
          if (!mbar_wait_warp(&q_empty[qs], ((t / Cfg::kQStages) & 1) ^ 1u, &cta_abort, p.status)) break;
          const long long at = ((static_cast<long long>(b) * p.H + h) * p.n_q + i) * BT;
          if (lead) {
            mbar_expect_tx(&q_full[qs], Cfg::kTileBytes + Cfg::kRowBytes);
#pragma unroll
            for (int hf = 0; hf < Cfg::kHalves; ++hf)
              tma_load_4d(sQ + qs * Cfg::kTileBytes + hf * 16384, &tmQ, &q_full[qs], hf * 64, i * BT, h, b);
            bulk_load(sRow + qs * Cfg::kRowBytes, p.lse2 + at, BT * 4, &q_full[qs]);
            bulk_load(sRow + qs * Cfg::kRowBytes + BT * 4, p.delta + at, BT * 4, &q_full[qs]);
          }
          if (!mbar_wait_warp(&do_empty[ds], ((t / Cfg::kDOStages) & 1) ^ 1u, &cta_abort, p.status)) break;
          if (lead) {
            mbar_expect_tx(&do_full[ds], Cfg::kTileBytes);
#pragma unroll
            for (int hf = 0; hf < Cfg::kHalves; ++hf)
              tma_load_4d(sDO + ds * Cfg::kTileBytes + hf * 16384, &tmDO, &do_full[ds], hf * 64, i * BT, h, b);
          }
          __syncwarp();
        }
      }
    } else if (warp == 13) {
      // ---------------------------------------------------------------- MMA issuer
      if (n_iter > 0) {
        const uint32_t lead = elect_one() ? 1u : 0u;
        constexpr uint32_t idesc_s = umma_idesc(BT, BT, 1, 1, 0, 0);   // S^T, dP^T: both operands K-major
        constexpr uint32_t idesc_kv = umma_idesc(BT, D, 1, 1, 0, 1);   // dV, dK: P^T / dS^T in TMEM, dO / Q N-major
        constexpr uint32_t idesc_q = umma_idesc(BT, D, 1, 1, 1, 1);    // dQ: dS M-major, K N-major
        const uint32_t k_base = smem_u32(sK), v_base = smem_u32(sV), ds_base = smem_u32(sDS);
        auto scores = [&](int t) -> bool {
          const int qs = t % Cfg::kQStages;
          if (!mbar_wait_warp(&q_full[qs], (t / Cfg::kQStages) & 1, &cta_abort, p.status)) return false;
          tc_fence_after();
          const uint32_t q_base = smem_u32(sQ + qs * Cfg::kTileBytes);
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            umma_f16_if(lead, tmem_base + Cfg::kColS, kmajor_desc<128>(k_base, ks), kmajor_desc<128>(q_base, ks), idesc_s, ks != 0);
          umma_commit_if(lead, &s_full);
          return true;
        };
        auto gradients_of_p = [&](int t) -> bool {     // dP^T = V dO^T
          const int ds = t % Cfg::kDOStages;
          if (!mbar_wait_warp(&do_full[ds], (t / Cfg::kDOStages) & 1, &cta_abort, p.status)) return false;
          // (with 128 columns dQ of the step before lies here)
          if (!Cfg::kOwnDQ && !mbar_wait_warp(&dq_read, (t & 1) ^ 1u, &cta_abort, p.status)) return false;
          tc_fence_after();
          const uint32_t do_base = smem_u32(sDO + ds * Cfg::kTileBytes);
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks)
            umma_f16_if(lead, tmem_base + Cfg::kColDP, kmajor_desc<128>(v_base, ks), kmajor_desc<128>(do_base, ks), idesc_s, ks != 0);
          umma_commit_if(lead, &dp_full);
          return true;
        };
        bool ok = mbar_wait_warp(&kv_full, 0, &cta_abort, p.status) && scores(0) && (!Cfg::kOwnDQ || gradients_of_p(0));
        for (int t = 0; ok && t < n_iter; ++t) {
          const uint32_t ph = t & 1;
          const uint32_t q_base = smem_u32(sQ + (t % Cfg::kQStages) * Cfg::kTileBytes);
          const uint32_t do_base = smem_u32(sDO + (t % Cfg::kDOStages) * Cfg::kTileBytes);
          if (!Cfg::kOwnDQ && !gradients_of_p(t)) break;
          if (!mbar_wait_warp(&p_full, ph, &cta_abort, p.status)) break;
          tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < BT / 16; ++ks)   // dV += P^T dO   (K = query rows; each half of P^T lies over its half of S^T)
            umma_f16_ts_if(lead, tmem_base + Cfg::kColDV, tmem_base + Cfg::kColS + (ks >> 2) * 64 + (ks & 3) * 8,
                           mnmajor_desc(do_base, ks, 16384), idesc_kv, (t | ks) != 0);
          umma_commit_if(lead, &do_empty[t % Cfg::kDOStages]);
          if (t + 1 < n_iter && !scores(t + 1)) break;
          if (!mbar_wait_warp(&ds_full, ph, &cta_abort, p.status)) break;
          tc_fence_after();
#pragma unroll
          for (int ks = 0; ks < BT / 16; ++ks)   // dK += dS^T Q
            umma_f16_ts_if(lead, tmem_base + Cfg::kColDK, tmem_base + Cfg::kColDP + (ks >> 2) * 64 + (ks & 3) * 8,
                           mnmajor_desc(q_base, ks, 16384), idesc_kv, (t | ks) != 0);
          umma_commit_if(lead, &q_empty[t % Cfg::kQStages]);
          if (Cfg::kOwnDQ) {
            if (t + 1 < n_iter && !gradients_of_p(t + 1)) break;
            if (!mbar_wait_warp(&dq_read, ph ^ 1u, &cta_abort, p.status)) break;
            tc_fence_after();
          }
#pragma unroll
          for (int ks = 0; ks < BT / 16; ++ks)   // dQ = dS K       (K = key rows; with 128 columns over dS^T, which dK has read)
            umma_f16_if(lead, tmem_base + Cfg::kColDQ, mnmajor_desc(ds_base, ks, 16384), mnmajor_desc(k_base, ks, 16384), idesc_q, ks != 0);
          umma_commit_if(lead, &dq_full);
        }
      }
    }
  } else if (warp >= 8) {
    // ---------------------------------------------------------------- dQ tiles -> fp32 scratch
    warpgroup_regs_inc<kBwdReduceRegs>();
    const uint32_t addr = tmem_base + (static_cast<uint32_t>((warp - 8) * 32) << 16) + Cfg::kColDQ;
    uint8_t* pieces = sPiece + (warp - 8) * Cfg::kPieces * Cfg::kPieceBytes;
    int piece = 0;
    Walk w = first;
    for (int t = 0; t < n_iter; ++t, next(w)) {
      const int at = w.i * BT + (warp - 8) * 32, rows = max(0, min(32, p.Sq - at));
      float* dst = p.dq_acc + ((static_cast<long long>(b) * p.H + w.h) * p.Sq + at) * D;
      // (TMEM accesses are warp-collective: a failed wait leaves the loop warp-uniformly)
      if (!__all_sync(0xffffffffu, mbar_wait(&dq_full, t & 1, &cta_abort, p.status) ? 1 : 0)) break;
      tc_fence_after();
      uint32_t r[D];                         // all of it at once: the tensor core waits for these columns
#pragma unroll
      for (int c = 0; c < D / 32; ++c) tmem_ld_32x32(addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&r[c * 32]));
      tmem_ld_wait();
      tc_fence_before();
      mbar_arrive(&dq_read);
      if (rows == 0) continue;
      if constexpr (Cfg::kPieces > 0) {
#pragma unroll
        for (int c = 0; c < D / 16; ++c) {
          uint8_t* buf = pieces + piece * Cfg::kPieceBytes;
          if (lane == 0) tma_store_wait_read<(Cfg::kPieces > 0 ? Cfg::kPieces - 1 : 0)>();          // the reduction that last read this buffer
          __syncwarp();
          if (lane < rows)
#pragma unroll
            for (int q = 0; q < 4; ++q)
              *reinterpret_cast<uint4*>(buf + (q * rows + lane) * 16) =
                  make_uint4(r[c * 16 + q * 4], r[c * 16 + q * 4 + 1], r[c * 16 + q * 4 + 2], r[c * 16 + q * 4 + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            bulk_add_f32(dst + c * 16 * rows, buf, rows * 64);
            tma_store_commit();
          }
          piece = piece == Cfg::kPieces - 1 ? 0 : piece + 1;
        }
      } else if (lane < rows) {
        dst += lane * 4;
#pragma unroll
        for (int e = 0; e < D; e += 4, dst += rows * 4)
          atomicAdd(reinterpret_cast<float4*>(dst),
                    make_float4(__uint_as_float(r[e]), __uint_as_float(r[e + 1]), __uint_as_float(r[e + 2]), __uint_as_float(r[e + 3])));
      }
    }
    if (Cfg::kPieces > 0 && lane == 0) tma_store_wait_all<0>();
  } else {
    // ---------------------------------------------------------------- P and dS (warps 0..7)
    warpgroup_regs_inc<kBwdComputeRegs>();
    const int half = warp >> 2, row = (warp & 3) * 32 + lane, key = c0 + row;      // query columns half * 64 ..
    const uint32_t lane_addr = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_addr = tmem_base + lane_addr + Cfg::kColS + half * 64, dp_addr = tmem_base + lane_addr + Cfg::kColDP + half * 64;
    uint8_t* ds_row = sDS + half * 16384 + row * 128;
    const float2 mul = make_float2(p.scale_log2, p.scale_log2);
    bool ok = true;
    Walk w = first;
    for (int t = 0; t < n_iter; ++t, next(w)) {
      const int q0 = w.i * BT;
      const uint32_t ph = t & 1;
      const float* lse = reinterpret_cast<const float*>(sRow + (t % Cfg::kQStages) * Cfg::kRowBytes) + half * 64;
      const float* delta = lse + BT;
      // lse before the wait for the scores, delta before the wait for dP: shared memory is busy with operands of MMAs, and
      // a load that is waited for takes long
      float4 l[16];
      bool here = mbar_wait(&q_full[t % Cfg::kQStages], (t / Cfg::kQStages) & 1, &cta_abort, p.status);
#pragma unroll
      for (int e = 0; e < 16; ++e) l[e] = reinterpret_cast<const float4*>(lse)[e];
      here = here && mbar_wait(&s_full, ph, &cta_abort, p.status);
      if (!__all_sync(0xffffffffu, here ? 1 : 0)) { ok = false; break; }
      tc_fence_after();
      float2 pr[32];
      auto probabilities = [&](auto masked, int from) {             // the columns from `from` on see the key
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t r[32], packed[16];
          tmem_ld_32x32(s_addr + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            const float4 l4 = l[c * 8 + e / 4];
            const float2 x = fma_f32x2(make_float2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])), mul,
                                       e & 2 ? make_float2(-l4.z, -l4.w) : make_float2(-l4.x, -l4.y));
            float2 y = make_float2(exp2_ftz(x.x), exp2_ftz(x.y));
            if constexpr (decltype(masked)::value) {
              if (c * 32 + e < from) y.x = 0.f;
              if (c * 32 + e + 1 < from) y.y = 0.f;
            }
            pr[c * 16 + e / 2] = y;
            packed[e / 2] = pack_bf16x2(y.x, y.y);
          }
          tmem_st_32x16(s_addr + c * 16, packed);
        }
      };
      if ((p.causal && c0 + BT - 1 > q0 + offset) || c0 + BT > p.Sk)
        probabilities(std::true_type{}, key >= p.Sk ? 64 : p.causal ? key - offset - q0 - half * 64 : 0);
      else
        probabilities(std::false_type{}, 0);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive(&p_full);
      float4 dl[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) dl[e] = reinterpret_cast<const float4*>(delta)[e];
      here = mbar_wait(&dp_full, ph, &cta_abort, p.status);
      // dQ of the step before has read dS in shared memory (its first pass finds the barrier open). Heads of 64 have no other wait for that: the dP
      // waited for above was issued in front of that dQ.
      here = here && mbar_wait(&dq_full, ph ^ 1u, &cta_abort, p.status);
      if (!__all_sync(0xffffffffu, here ? 1 : 0)) { ok = false; break; }
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32], packed[16];
        tmem_ld_32x32(dp_addr + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 32; e += 2) {
          const float4 d4 = dl[e / 4];
          const float2 d = add_f32x2(make_float2(__uint_as_float(r[e]), __uint_as_float(r[e + 1])),
                                     e & 2 ? make_float2(-d4.z, -d4.w) : make_float2(-d4.x, -d4.y));
          const float2 x = mul_f32x2(pr[c * 16 + e / 2], d);
          packed[e / 2] = pack_bf16x2(x.x, x.y);
        }
        tmem_st_32x16(dp_addr + c * 16, packed);
        if (c == 0)
#pragma unroll
          for (int e = 0; e < 8; ++e) dl[e] = reinterpret_cast<const float4*>(delta)[8 + e];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          *reinterpret_cast<uint4*>(ds_row + (((c * 4 + q) ^ (row & 7)) << 4)) =
              make_uint4(packed[q * 4], packed[q * 4 + 1], packed[q * 4 + 2], packed[q * 4 + 3]);
      }
      tmem_st_wait();
      tc_fence_before();
      fence_proxy_async_smem();
      mbar_arrive(&ds_full);
    }
    // ---------------------------------------------------------------- dK (warps 0-3), dV (warps 4-7) out
    bool have = ok && n_iter > 0;
    if (have) have = mbar_wait(&dq_full, (n_iter - 1) & 1, &cta_abort, p.status);   // (covers every MMA issued before it)
    have = __all_sync(0xffffffffu, have ? 1 : 0) != 0;
    if (have || n_iter == 0) {
      if (have) tc_fence_after();
      // K and V are not needed any more: their shared memory turns the rows, so that a warp stores whole rows
      uint8_t* tile = half ? sV : sK;
      const float f = half ? 1.f : p.scale;
#pragma unroll 1
      for (int c = 0; c < D / 32; ++c) {
        uint32_t r[32];
        if (have) {
          tmem_ld_32x32(tmem_base + lane_addr + (half ? Cfg::kColDV : Cfg::kColDK) + c * 32, r);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0u;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint4 v;
          v.x = pack_bf16x2(__uint_as_float(r[q * 8]) * f, __uint_as_float(r[q * 8 + 1]) * f);
          v.y = pack_bf16x2(__uint_as_float(r[q * 8 + 2]) * f, __uint_as_float(r[q * 8 + 3]) * f);
          v.z = pack_bf16x2(__uint_as_float(r[q * 8 + 4]) * f, __uint_as_float(r[q * 8 + 5]) * f);
          v.w = pack_bf16x2(__uint_as_float(r[q * 8 + 6]) * f, __uint_as_float(r[q * 8 + 7]) * f);
          *reinterpret_cast<uint4*>(tile + (c >> 1) * 16384 + row * 128 + ((((c & 1) * 4 + q) ^ (row & 7)) << 4)) = v;
        }
      }
      __syncwarp();
      constexpr int kChunks = D / 8, kRows = 32 / kChunks;       // 16-byte chunks per row, rows per store
      __nv_bfloat16* out = (half ? p.dv : p.dk) + b * p.sb + hk * p.sh;
      const int ch = lane % kChunks;
#pragma unroll 4
      for (int i = 0; i < 32; i += kRows) {
        const int r = (warp & 3) * 32 + i + lane / kChunks;
        const uint4 v = *reinterpret_cast<const uint4*>(tile + (ch >> 3) * 16384 + r * 128 + (((ch & 7) ^ (r & 7)) << 4));
        if (c0 + r < p.Sk) *reinterpret_cast<uint4*>(out + static_cast<long long>(c0 + r) * p.ss + ch * 8) = v;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 13) {
    if (cta_abort) {
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Per row of [B, H, n_q * 128]: lse2 = lse * log2 e and delta = sum_d dO * O (both [B, Sq, H, D], contiguous), and the row's share
// of the zeroes of dq_acc. D / 8 lanes take a row, 16 bytes each; an O whose base is not aligned to that is read by elements.
template <int D>
__global__ void __launch_bounds__(256)
flash_bwd_rows_kernel(const __nv_bfloat16* __restrict__ dO, const __nv_bfloat16* __restrict__ O, const float* __restrict__ lse,
                      float* __restrict__ lse2, float* __restrict__ delta, float* __restrict__ dq_acc, long long rows, int Sq, int Sp, int H) {
  constexpr int kLanes = D / 8;
  const long long at = (blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x) / kLanes;      // row of [B, H, Sp]
  const int c = threadIdx.x % kLanes;
  if (at >= rows) return;                       // (rows is a multiple of 128: whole warps leave)
  const long long bh = at / Sp;
  const int s = static_cast<int>(at - bh * Sp);
  float acc = 0.f;
  if (s < Sq) {
    const long long b = bh / H, src = ((b * Sq + s) * H + (bh - b * H)) * D + c * 8;
    const uint4 x = *reinterpret_cast<const uint4*>(dO + src);
    uint4 y;
    if ((reinterpret_cast<uintptr_t>(O) & 15) == 0) {
      y = *reinterpret_cast<const uint4*>(O + src);
    } else {
      const unsigned short* e = reinterpret_cast<const unsigned short*>(O + src);
      y = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
    }
    const __nv_bfloat162 *x2 = reinterpret_cast<const __nv_bfloat162*>(&x), *y2 = reinterpret_cast<const __nv_bfloat162*>(&y);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 u = __bfloat1622float2(x2[i]), v = __bfloat1622float2(y2[i]);
      acc = fmaf(u.x, v.x, fmaf(u.y, v.y, acc));
    }
    float4* z = reinterpret_cast<float4*>(dq_acc + (bh * Sq + s) * D + c * 8);
    z[0] = z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int o = kLanes / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (c == 0) {
    const float l = s < Sq ? lse[bh * Sq + s] : -INFINITY;
    lse2[at] = l == -INFINITY ? INFINITY : l * 1.4426950408889634f;
    delta[at] = acc;
  }
}

// dq[b, s, h, :] (bf16, strided) = scale * dq_acc. A warp takes 32 rows: lane = row % 8 + 8 * (eight columns).
template <int D>
__global__ void __launch_bounds__(128)
flash_bwd_dq_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dq, float scale, int H, int Sq, long long sb, long long ss,
                    long long sh) {
  const int lane = threadIdx.x & 31, s0 = blockIdx.x * BT + (threadIdx.x >> 5) * 32, h = blockIdx.y, b = blockIdx.z;
  const int rows = min(32, Sq - s0);
  const float* src = acc + ((static_cast<long long>(b) * H + h) * Sq + s0) * D;
  __nv_bfloat16* out = dq + b * sb + static_cast<long long>(s0) * ss + h * sh;
  for (int r = lane & 7; r < rows; r += 8) {
#pragma unroll
    for (int c = lane >> 3; c < D / 8; c += 4) {
      const float4 x = *reinterpret_cast<const float4*>(src + (2 * c * rows + r) * 4);
      const float4 y = *reinterpret_cast<const float4*>(src + ((2 * c + 1) * rows + r) * 4);
      uint4 v;
      v.x = pack_bf16x2(x.x * scale, x.y * scale);
      v.y = pack_bf16x2(x.z * scale, x.w * scale);
      v.z = pack_bf16x2(y.x * scale, y.y * scale);
      v.w = pack_bf16x2(y.z * scale, y.w * scale);
      *reinterpret_cast<uint4*>(out + r * ss + c * 8) = v;
    }
  }
}

}  // namespace
}  // namespace tsb

// Bytes of fp32 scratch tsb_flash_bwd needs: the dQ accumulator [B, Sq, H, D], then lse2 and delta [B, H, Sq rounded up to 128].
TSB_EXPORT long long tsb_flash_bwd_scratch_bytes(int B, int Sq, int H, int D) {
  const long long Sp = (Sq + 127) / 128 * 128;
  return (static_cast<long long>(B) * Sq * H * D + 2 * static_cast<long long>(B) * H * Sp) * 4;
}

// Gradients of tsb_flash_fwd. dO and O are contiguous [B, Sq, H, D], dO, q, k and v 16-byte aligned. dq / dk / dv are bf16 views that share the stride triple
// (g_sb, g_ss, g_sh) -- usually slices of one packed [B, S, H + 2 Hkv, D] buffer.
// scratch: tsb_flash_bwd_scratch_bytes() bytes of device memory, 16-byte aligned (contents are overwritten).
TSB_EXPORT int tsb_flash_bwd(const void* dO, const void* q, const void* k, const void* v, const void* o,
                             const float* lse, void* dq, void* dk, void* dv, void* scratch, int B, int Sq, int Sk,
                             int H, int Hkv, int D, long long q_sb, long long q_ss, long long q_sh, long long k_sb,
                             long long k_ss, long long k_sh, long long v_sb, long long v_ss, long long v_sh,
                             long long g_sb, long long g_ss, long long g_sh, float scale, int causal, void* stream) {
  using namespace tsb;
  if (B <= 0 || Sq <= 0 || Sk <= 0 || H <= 0 || Hkv <= 0 || H % Hkv || (D != 64 && D != 128)) return -2;
  if (!scratch || (reinterpret_cast<uintptr_t>(scratch) & 15)) return -2;
  const long long strides[] = {q_sb, q_ss, q_sh, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh, g_sb, g_ss, g_sh};
  for (long long s : strides)
    if (s % 8) return -2;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long long c_sh = D, c_ss = static_cast<long long>(H) * D, c_sb = c_ss * Sq;
  const int n_q = (Sq + BT - 1) / BT;
  const long long rows = static_cast<long long>(B) * H * n_q * BT;
  float* dq_acc = static_cast<float*>(scratch);
  float* lse2 = dq_acc + static_cast<long long>(B) * Sq * H * D;
  float* delta = lse2 + rows;
  CUtensorMap tq, tk, tv, tdo;
  if (!make_bshd_tmap(&tq, q, B, Sq, H, D, q_sb, q_ss, q_sh, 128)) return -3;
  if (!make_bshd_tmap(&tk, k, B, Sk, Hkv, D, k_sb, k_ss, k_sh, 128)) return -3;
  if (!make_bshd_tmap(&tv, v, B, Sk, Hkv, D, v_sb, v_ss, v_sh, 128)) return -3;
  if (!make_bshd_tmap(&tdo, dO, B, Sq, H, D, c_sb, c_ss, c_sh, 128)) return -3;
  BwdParams p;
  p.lse2 = lse2;
  p.delta = delta;
  p.dq_acc = dq_acc;
  p.dk = static_cast<__nv_bfloat16*>(dk);
  p.dv = static_cast<__nv_bfloat16*>(dv);
  p.Sq = Sq; p.Sk = Sk; p.H = H; p.Hkv = Hkv; p.n_q = n_q;
  p.sb = g_sb; p.ss = g_ss; p.sh = g_sh;
  p.scale = scale;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal;
  p.status = device_status_word();
  auto go = [&](auto dim, auto kern, auto rows_kern, auto dq_kern) -> int {
    constexpr int kD = decltype(dim)::value;
    static PerDeviceFlag attr_set;                      // (one per D)
    cudaError_t e = cudaSuccess;
    if (attr_set.unset()) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, BwdCfg<kD>::kSmemBytes);
      if (e != cudaSuccess) return static_cast<int>(e);
      attr_set.set();
    }
    rows_kern<<<static_cast<unsigned>((rows * (kD / 8) + 255) / 256), 256, 0, s>>>(
        static_cast<const __nv_bfloat16*>(dO), static_cast<const __nv_bfloat16*>(o), lse, lse2, delta, dq_acc, rows, Sq, n_q * BT, H);
    kern<<<dim3(static_cast<unsigned>(Hkv) * ((Sk + BT - 1) / BT), 1, B), kBwdThreads, BwdCfg<kD>::kSmemBytes, s>>>(tq, tk, tv, tdo, p);
    e = cudaGetLastError();
    if (e != cudaSuccess) return static_cast<int>(e);
    dq_kern<<<dim3(n_q, H, B), 128, 0, s>>>(dq_acc, static_cast<__nv_bfloat16*>(dq), scale, H, Sq, g_sb, g_ss, g_sh);
    return static_cast<int>(cudaGetLastError());
  };
  return D == 128 ? go(std::integral_constant<int, 128>{}, flash_bwd_kernel<128>, flash_bwd_rows_kernel<128>, flash_bwd_dq_kernel<128>)
                  : go(std::integral_constant<int, 64>{}, flash_bwd_kernel<64>, flash_bwd_rows_kernel<64>, flash_bwd_dq_kernel<64>);
}
