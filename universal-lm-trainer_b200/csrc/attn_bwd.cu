// Causal FlashAttention-2 backward for head_dim 64 on sm_100a.
//
// Replaces fa_bwd of the reference (csrc/flash_attn_v100/flash_attn_v100_bwd.cu:
// delta pre-pass :42-61, dQ kernel :66-219, dK/dV kernel :224-428) with the same
// three-kernel split and the same formulas (flash_attn_v100_bwd.cu:10-15):
//   P = exp2(S*scale*log2e - lse*log2e),  P_d = keep * P / (1-p),
//   delta = rowsum(O * dO),  dP = dO V^T,  dS = P_d * dP - P * delta,
//   dV = P_d^T dO,  dQ = scale * dS K,  dK = scale * dS^T Q,
// P and dS rounded to the 16-bit type before their MMAs.
//
// Machine mapping (both tensor-core kernels): TMA-staged 128-byte-swizzled
// tiles, tcgen05.mma with fp32 accumulators in TMEM, the 16-bit P / dS operands
// written back into TMEM and consumed as the A operand, so no intermediate
// ever touches shared or global memory.
//   dQ kernel:   CTA = 128 query rows (compute thread r = row r = TMEM lane r),
//                walks key tiles of 64: S and dP (128x64 each) -> dS -> dQ += dS K.
//   dK/dV kernel: CTA = 128 keys (thread r = key r), walks query tiles of 64 from
//                the diagonal down, transposed view: S^T = K Q^T, dP^T = V dO^T,
//                dV += P^T dO, dK += dS^T Q.
// In both a thread owns a row: it takes the tile's S and dP of its row into registers and releases their TMEM columns at
// once, and P / dS go to columns of their own, so no tile waits for the round trip "P / dS written -> gradient MMAs -> columns
// free -> scores".  Two warps of compute share a scheduler (two CTAs in the dQ kernel, two groups in the dK/dV kernel).  Each
// accumulator has exactly one issuing thread, so the summation order, and with it the result, is the same on every run.  All
// barrier waits are bounded (status bit + clean exit on expiry); the compute warps make the outcome of a wait warp-uniform
// by a vote, because warp-wide TMEM loads follow.
//
// Fused RoPE adjoint (template parameter ROPE): q and k are the rotated tensors; the
// dQ and dK epilogues round their result to 16 bits, hand the accumulator back, and
// then apply the adjoint rotation (rope_math.cuh: the stand-alone kernel's arithmetic
// on the same 16-bit values, so the bits are equal) before the one store each row
// gets anyway -- the separate RoPE-backward launch and its read+write of dQ and dK
// disappear.
#include <type_traits>

#include "tc.cuh"
#include "rope_math.cuh"

namespace ulm {
namespace {

using namespace tc;

constexpr int HD = 64;
constexpr int BR = 128;                 // rows owned by a CTA (queries or keys)
constexpr int BT = 64;                  // rows of the streamed tile
constexpr int kGroups = 2;              // dK/dV kernel: compute groups; tile t is worked on by group t % kGroups, in that group's TMEM columns
constexpr int kGroupWarps = 4, kGroupThreads = 32 * kGroupWarps;   // a thread per row of the tile
constexpr int kStages = 6;              // dK/dV kernel: streamed-tile ring
static_assert(192 * kGroups + 128 <= 512, "score buffers, packed operands and accumulators must fit 512 TMEM columns");
// The other roles of the dK/dV kernel, one warp each, after the compute warps: TMA producer, the S issuer, the dP issuer and the
// gradient issuer (dV and dK); then the warpgroup that writes finished gradients out.
constexpr int kProducerWarp = kGroupWarps * kGroups, kMmaWarp = kProducerWarp + 1, kMma2Warp = kProducerWarp + 2, kGradWarp = kProducerWarp + 3,
              kStoreWarp = kProducerWarp + 4;
constexpr int kThreadsKV = 32 * (kStoreWarp + 4);
// Per thread, by warpgroup.  The plain kernels spill 100-170 bytes all the same, the ones with the RoPE adjoint 370-410: there a storing
// thread holds both rounded rows (64 registers) beside the tables' values (64).  168 / 56 / 120, 176 / 56 / 104 and 200 / 40 / 72
// were slower.
constexpr int kRegsCompute = 184, kRegsIssue = 56, kRegsStore = 88;
static_assert(kGroups * kGroupThreads * kRegsCompute + 128 * (kRegsIssue + kRegsStore) <= 65536 / kThreadsKV / 8 * 8 * kThreadsKV,
              "the register split must fit what the CTA is launched with");
constexpr uint32_t kBigTile = BR * HD * 2;    // 16 KB
constexpr uint32_t kSmallTile = BT * HD * 2;  //  8 KB
constexpr uint32_t kTmemCols = 512;
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ uint32_t hash_u32(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352dU;
  x ^= x >> 15; x *= 0x846ca68bU;
  x ^= x >> 16;
  return x;
}
// keep mask of the reference (fa_common.cuh:30-38)
__device__ __forceinline__ bool dropout_keep(uint32_t seed_mix, int row, int col, float p) {
  uint32_t h = seed_mix ^ ((uint32_t)(row + 1) * 0x85EBCA6Bu) ^ ((uint32_t)(col + 1) * 0xC2B2AE35u);
  h = hash_u32(h);
  return ((h >> 8) * (1.0f / 16777216.0f)) >= p;
}

// dS of two neighbouring score elements without dropout, two-wide fp32 arithmetic (one issue slot per pair, same
// rounding as the scalar operations): p = 2^(s*scale2 - lse2), dS = p * (dP - delta); nl and nd hold the NEGATED
// statistics of the two elements.  keep(e) says whether element e is inside the mask.
template <typename Keep>
__device__ __forceinline__ void pair_ds(uint32_t s0, uint32_t s1, uint32_t dp0, uint32_t dp1, uint64_t sc2, uint64_t nl, uint64_t nd,
                                        Keep keep, float (&d)[2], float* p_out = nullptr) {
  float x0, x1;
  f2_unpack(f2_fma(f2_pack(__uint_as_float(s0), __uint_as_float(s1)), sc2, nl), x0, x1);
  float p0 = ex2_ordered(x0), p1 = ex2_ordered(x1);
  p0 = keep(0) ? p0 : 0.f;
  p1 = keep(1) ? p1 : 0.f;
  if (p_out) { p_out[0] = p0; p_out[1] = p1; }
  f2_unpack(f2_mul(f2_pack(p0, p1), f2_add(f2_pack(__uint_as_float(dp0), __uint_as_float(dp1)), nd)), d[0], d[1]);
}

template <typename T> struct Fmt { static constexpr int v = 0; };
template <> struct Fmt<__nv_bfloat16> { static constexpr int v = 1; };

// The four warps that share a staging tile (the dQ kernel's compute warps, the dK/dV kernel's storing warps)
__device__ __forceinline__ void quad_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }

// All lanes of a warp learn together whether the wait succeeded.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag));
}

// The threads of those four warps learn together whether any of them says yes.
__device__ __forceinline__ bool quad_any(bool yes) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 q, %1, 0;\n\t"
      "bar.red.or.pred p, 1, 128, q;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(any) : "r"((uint32_t)yes) : "memory");
  return any != 0;
}

// Four floats from shared memory, kept in program order with respect to other such calls and the exponentials
__device__ __forceinline__ void lds_f4(const float* p, float* v) {
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(smem_u32(p)) : "memory");
}

// Tables of the fused RoPE adjoint (unused when ROPE is false).
struct RopeTab {
  const float* cos_tab; const float* sin_tab;
  int64_t cos_stride, sin_stride;
};

// 32 accumulator columns of this thread's row, scaled and rounded to 16 bits: four 16-byte vectors
template <typename T>
__device__ __forceinline__ void acc_to_16bit(uint32_t taddr, float f, uint4 (&out)[4]) {
  uint32_t ov[32];
  tmem_ld32(taddr, ov);
  tmem_wait_ld();
#pragma unroll
  for (int v4 = 0; v4 < 4; ++v4) {
    out[v4].x = Cvt<T>::pack2(__uint_as_float(ov[v4 * 8 + 0]) * f, __uint_as_float(ov[v4 * 8 + 1]) * f);
    out[v4].y = Cvt<T>::pack2(__uint_as_float(ov[v4 * 8 + 2]) * f, __uint_as_float(ov[v4 * 8 + 3]) * f);
    out[v4].z = Cvt<T>::pack2(__uint_as_float(ov[v4 * 8 + 4]) * f, __uint_as_float(ov[v4 * 8 + 5]) * f);
    out[v4].w = Cvt<T>::pack2(__uint_as_float(ov[v4 * 8 + 6]) * f, __uint_as_float(ov[v4 * 8 + 7]) * f);
  }
}

// ---------------------------------------------------------------------------
// Fused RoPE adjoint of a 128-row gradient tile held one row per thread by four warps.
// A thread that owned a row would have to read its own table row: 32 different 128-byte lines per warp
// load, which makes the load/store unit the cost.  So the rounded 16-bit rows go through a small shared
// staging tile (64 rows x 128 bytes, 128-byte swizzle) and are picked up again with
// eight threads per row (rope_math.cuh): table loads and the final global stores are then fully
// coalesced.  Two passes of 64 rows; the tables of pass 0 are prefetched into registers before the wait
// for the accumulator (see the callers), those of pass 1 while pass 0 is being worked on.
// ---------------------------------------------------------------------------
constexpr int kRopeStageRows = 64;
constexpr uint32_t kRopeStageBytes = kRopeStageRows * 128;
constexpr int kRopeTasks = kRopeStageRows * 8 / 128;                // per thread and pass

__device__ __forceinline__ void rope_prefetch_pass(RopeQuad (&tab)[kRopeTasks], const RopeTab& rt, int row0, int pass, int tg, int S) {
#pragma unroll
  for (int j = 0; j < kRopeTasks; ++j) {
    const int idx = j * 128 + tg;
    const int row = row0 + kRopeStageRows * pass + (idx >> 3);
    const int pos = row < S ? row : S - 1;
    rope_load_quad(tab[j], rt.cos_tab + (int64_t)pos * rt.cos_stride, rt.sin_tab + (int64_t)pos * rt.sin_stride, idx & 7);
  }
}

// `lo` / `hi`: columns [0,32) / [32,64) of this thread's row r.  `item_out` points at row 0 of the item in the output tensor.
template <typename T>
__device__ __forceinline__ void rope_adjoint_store(uint8_t* stage, int tg, int r, const uint4 (&lo)[4], const uint4 (&hi)[4],
                                                   T* item_out, int64_t row_stride, int row0, int S, const RopeTab& rt,
                                                   RopeQuad (&tab)[kRopeTasks]) {
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    if ((r >> 6) == pass) {
      const int rr = r & 63;
      uint8_t* srow = stage + rr * 128;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        *reinterpret_cast<uint4*>(srow + ((c ^ (rr & 7)) << 4)) = lo[c];
        *reinterpret_cast<uint4*>(srow + (((4 + c) ^ (rr & 7)) << 4)) = hi[c];
      }
    }
    quad_sync();
#pragma unroll
    for (int j = 0; j < kRopeTasks; ++j) {
      const int idx = j * 128 + tg;
      const int row = idx >> 3, cg = idx & 7;
      const uint2 glo = *reinterpret_cast<const uint2*>(stage + swz_quad_offset(row, cg));
      const uint2 ghi = *reinterpret_cast<const uint2*>(stage + swz_quad_offset(row, cg + 8));
      uint2 olo, ohi;
      rope_apply_quad<T, true>(tab[j], glo, ghi, olo, ohi);
      const int trow = kRopeStageRows * pass + row;
      if (row0 + trow < S) {
        T* dst = item_out + (int64_t)trow * row_stride;
        *reinterpret_cast<uint2*>(dst + 4 * cg) = olo;
        *reinterpret_cast<uint2*>(dst + 32 + 4 * cg) = ohi;
      }
    }
    if (pass == 0) rope_prefetch_pass(tab, rt, row0, 1, tg, S);
    quad_sync();                                    // the tile is rewritten by the next pass / the next epilogue
  }
}

// The plain store of a gradient tile held one row per thread: each warp passes its 32 rows through 4 KB of its own, so that the
// stores are coalesced whatever the layout (a thread that wrote its own row would spread every store instruction over 32 lines).
constexpr uint32_t kWarpStageBytes = 32 * 128;
template <typename T>
__device__ __forceinline__ void staged_store(uint8_t* stage, int lane, const uint4 (&lo)[4], const uint4 (&hi)[4], T* warp_out,
                                             int64_t row_stride, int rows) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    *reinterpret_cast<uint4*>(stage + lane * 128 + ((c ^ (lane & 7)) << 4)) = lo[c];
    *reinterpret_cast<uint4*>(stage + lane * 128 + (((4 + c) ^ (lane & 7)) << 4)) = hi[c];
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int row = i * 4 + (lane >> 3), c = lane & 7;
    const uint4 u = *reinterpret_cast<const uint4*>(stage + row * 128 + ((c ^ (row & 7)) << 4));
    if (row < rows) *reinterpret_cast<uint4*>(warp_out + (int64_t)row * row_stride + c * 8) = u;
  }
  __syncwarp();                                           // the rows are rewritten by the next store
}

// ---------------------------------------------------------------------------
// delta[bh, s] = sum_d O[s, d] * dO[s, d]   (fp32), 8 threads per row
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
attn_delta_kernel(const T* __restrict__ O, const T* __restrict__ dO, float* __restrict__ delta,
                  int64_t o_sb, int64_t o_sh, int64_t o_ss, int64_t do_sb, int64_t do_sh, int64_t do_ss,
                  int S, int H) {
  const int part = threadIdx.x & 7;
  const int row = blockIdx.x * 32 + (threadIdx.x >> 3);
  const int bh = blockIdx.y, b = bh / H, h = bh % H;
  float sum = 0.f;
  if (row < S) {
    const uint4 ov = *reinterpret_cast<const uint4*>(O + b * o_sb + h * o_sh + (int64_t)row * o_ss + part * 8);
    const uint4 gv = *reinterpret_cast<const uint4*>(dO + b * do_sb + h * do_sh + (int64_t)row * do_ss + part * 8);
    const uint32_t* ow = reinterpret_cast<const uint32_t*>(&ov);
    const uint32_t* gw = reinterpret_cast<const uint32_t*>(&gv);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 a = Cvt<T>::unpack2(ow[i]), g = Cvt<T>::unpack2(gw[i]);
      sum += a.x * g.x + a.y * g.y;
    }
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);
  sum += __shfl_xor_sync(0xffffffffu, sum, 2);
  sum += __shfl_xor_sync(0xffffffffu, sum, 4);
  if (part == 0 && row < S) delta[(int64_t)bh * S + row] = sum;
}

// ---------------------------------------------------------------------------
// dQ kernel
// One CTA per work item (128 query rows of one (batch, head)), two CTAs per SM, so that one CTA's exponentials run
// under the other's waits, loads and stores, and a CTA's start-up and epilogue under the other's tiles.
// TMEM columns: S at 0, dP at 64, packed dS at 128, the dQ accumulator at 192.  A compute thread owns a query row: it takes the
// 64 + 64 values of its row into registers and hands both buffers back at once, so the next tile's S and dP are
// there when it has written this tile's dS, into columns that the previous tile's gradient MMAs have long read.
// What bounds it: the SFU (64 exponentials a thread and tile; 61 % of its peak at B8 H12 S4096, tensor pipe 45 %, issue slots
// 41 %), then the synchronisation around a tile, whose instructions queue behind the exponentials.  Against one persistent CTA per SM
// with three score buffer pairs, which waited a round trip through the tensor core for every pair, on one GPU (us): B8 H12 S4096 bf16
// 371 -> 335, B24 H12 S1363 fp16 179 -> 162, B4 H12 S201 8.6 -> 7.5, B1 H12 S67 6.6 -> 5.8, B64 H12 S300 64 -> 64, B1 H16 S4096
// 69 -> 70.5 (512 CTAs are not quite two waves).
// ---------------------------------------------------------------------------
constexpr int kStagesQ = 3;                // K/V tile ring
constexpr int kThreadsQ = 32 * (4 + 2);    // compute warps, producer warp, MMA warp
struct CtlQ {
  uint64_t qdo_full, kv_full[kStagesQ], kv_empty[kStagesQ], sdp_full, sdp_free, ds_ready, dq_done;
  uint32_t tmem_base;
  int abort;
  uint32_t fail_bits;
};
constexpr uint32_t kTmemColsQ = 256, kColDP = 64, kColDS = 128, kColDQ = 192;
constexpr size_t kSmemQ = 1024 + 3 * (size_t)kBigTile + (size_t)kStagesQ * 2 * kSmallTile + sizeof(CtlQ);

// FUSE_DELTA: the kernel also loads the item's O tile, computes delta = rowsum(O * dO) for its 128 rows
// itself and writes it to DELTA for the dK/dV kernel that follows on the stream; otherwise DELTA is an input.
template <typename T, bool CAUSAL, bool DROPOUT, bool FUSE_DELTA, bool ROPE>
__global__ void __launch_bounds__(kThreadsQ, 2)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                   const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                   const __grid_constant__ CUtensorMap tmO,
                   const float* __restrict__ LSE, float* __restrict__ DELTA, T* __restrict__ dQ,
                   int64_t dq_sb, int64_t dq_sh, int64_t dq_ss, int S, int H, float scale, float scale2,
                   float dropout_p, uint32_t seed, uint32_t* status, const RopeTab rt) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = base;                                    // dQ is staged here once the scores are done
  uint8_t* sdO = base + kBigTile;
  uint8_t* sO = base + 2 * kBigTile;
  uint8_t* sKV = base + 3 * kBigTile;                    // [stage][K|V], 8 KB each
  CtlQ* ctl = reinterpret_cast<CtlQ*>(sKV + (size_t)kStagesQ * 2 * kSmallTile);
  volatile int* abort_flag = &ctl->abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bh = blockIdx.x, b = bh / H, h = bh - b * H;
  const int qt = (int)gridDim.y - 1 - (int)blockIdx.y;   // the last query tile is the heaviest under the causal mask: scheduled first
  const int m0 = qt * BR;
  const int n_all = (S + BT - 1) / BT;
  const int n_causal = (m0 + BR) / BT;
  const int nkv = CAUSAL ? (n_causal < n_all ? n_causal : n_all) : n_all;

  if (threadIdx.x == 0) {
    mbar_init(&ctl->qdo_full, 1);
    for (int s = 0; s < kStagesQ; ++s) { mbar_init(&ctl->kv_full[s], 1); mbar_init(&ctl->kv_empty[s], 1); }
    mbar_init(&ctl->sdp_full, 1);
    mbar_init(&ctl->sdp_free, 4);
    mbar_init(&ctl->ds_ready, 4);
    mbar_init(&ctl->dq_done, 1);
    ctl->abort = 0;
    ctl->fail_bits = 0;
    fence_mbar_init();
  }
  if (warp == 5) { tmem_alloc(&ctl->tmem_base, kTmemColsQ); tmem_relinquish(); }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);   // warp-uniform

  if (warp == 4) {
    // ------------------------------ TMA producer ------------------------------
    if (elect_one()) {
      tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO);
      if (FUSE_DELTA) tma_prefetch_desc(&tmO);
      mbar_expect_tx(&ctl->qdo_full, (FUSE_DELTA ? 3 : 2) * kBigTile);
      tma_load_4d(sQ, &tmQ, &ctl->qdo_full, 0, m0, h, b);
      tma_load_4d(sdO, &tmdO, &ctl->qdo_full, 0, m0, h, b);
      if (FUSE_DELTA) tma_load_4d(sO, &tmO, &ctl->qdo_full, 0, m0, h, b);
      int j = 0;
      for (; j < nkv; ++j) {
        const int s = j % kStagesQ;
        if (j >= kStagesQ && !mbar_wait(&ctl->kv_empty[s], ((j / kStagesQ) - 1) & 1, abort_flag)) { atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_MMA); break; }
        uint8_t* dst = sKV + (size_t)s * 2 * kSmallTile;
        mbar_expect_tx(&ctl->kv_full[s], 2 * kSmallTile);
        tma_load_4d(dst, &tmK, &ctl->kv_full[s], 0, j * BT, h, b);
        tma_load_4d(dst + kSmallTile, &tmV, &ctl->kv_full[s], 0, j * BT, h, b);
      }
      if (*abort_flag) {   // let our own copies land before the CTA's shared memory goes away
        auto drain = [](uint64_t* full, uint32_t parity) {
          const uint64_t t0 = globaltimer_ns();
          while (!mbar_try(full, parity))
            if (globaltimer_ns() - t0 > kWaitLimitNs) break;
        };
        drain(&ctl->qdo_full, 0);
        for (int u = j > kStagesQ ? j - kStagesQ : 0; u < j; ++u) drain(&ctl->kv_full[u % kStagesQ], (u / kStagesQ) & 1);
      }
    }
  } else if (warp == 5) {
    // ------------------------------ MMA issuer --------------------------------
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc(Fmt<T>::v, BR, BT, 0);   // 128 x 64, both K-major
      constexpr uint32_t idesc_q = make_idesc(Fmt<T>::v, BR, HD, 1);   // 128 x 64, B = K tile read MN-major
      bool ok = mbar_wait(&ctl->qdo_full, 0, abort_flag);
      if (!ok) atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_LOAD);
      const uint64_t dq = make_sdesc_sw128(smem_u32(sQ)), ddo = make_sdesc_sw128(smem_u32(sdO));
      auto issue_scores = [&](int j) -> bool {             // S_j = Q K_j^T, dP_j = dO V_j^T
        const int s = j % kStagesQ;
        if (!mbar_wait(&ctl->kv_full[s], (j / kStagesQ) & 1, abort_flag)) { atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_LOAD); return false; }
        fence_after_sync();
        const uint64_t dk = make_sdesc_sw128(smem_u32(sKV + (size_t)s * 2 * kSmallTile)), dv = dk + (kSmallTile >> 4);
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) mma_ss(tmem_base, dq + (uint64_t)(kk * 2), dk + (uint64_t)(kk * 2), idesc_s, kk > 0);
#pragma unroll
        for (int kk = 0; kk < HD / 16; ++kk) mma_ss(tmem_base + kColDP, ddo + (uint64_t)(kk * 2), dv + (uint64_t)(kk * 2), idesc_s, kk > 0);
        mma_commit(&ctl->sdp_full);
        return true;
      };
      if (ok) ok = issue_scores(0);
      for (int j = 0; ok && j < nkv; ++j) {
        const int s = j % kStagesQ;
        if (j + 1 < nkv) {                                 // the compute warps free S and dP long before they have this tile's dS
          if (!mbar_wait(&ctl->sdp_free, j & 1, abort_flag)) { atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_SOFTMAX); break; }
          if (!issue_scores(j + 1)) break;
        }
        if (!mbar_wait(&ctl->ds_ready, j & 1, abort_flag)) { atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_SOFTMAX); break; }
        fence_after_sync();
        const uint64_t dk = make_sdesc_sw128(smem_u32(sKV + (size_t)s * 2 * kSmallTile));
#pragma unroll
        for (int kk = 0; kk < BT / 16; ++kk)               // 16 keys = 2048 bytes of K, 8 TMEM columns of dS
          mma_ts(tmem_base + kColDQ, tmem_base + kColDS + (uint32_t)(kk * 8), dk + (uint64_t)(kk * (2048 >> 4)), idesc_q, (j > 0 || kk > 0) ? 1u : 0u);
        mma_commit(&ctl->dq_done);
        mma_commit(&ctl->kv_empty[s]);
      }
    }
  } else {
    // ------------------------------ compute warps -----------------------------
    const int r = warp * 32 + lane;                      // query row within the tile == TMEM lane
    const int grow = m0 + r;
    const uint32_t t_row = tmem_base + ((uint32_t)(warp * 32) << 16);
    const uint32_t seed_mix = (seed * 0x9E3779B1u) ^ (((uint32_t)bh + 1u) * 0x27D4EB2Fu);
    const float inv_keep = DROPOUT ? 1.f / (1.f - dropout_p) : 1.f;
    const float lse2 = grow < S ? LSE[(int64_t)bh * S + grow] * kLog2e : INFINITY;
    bool ok = true;
    float dlt = 0.f;
    if (FUSE_DELTA) {
      ok = warp_wait(&ctl->qdo_full, 0, abort_flag);
      if (!ok && lane == 0) atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_LOAD);
      if (ok) {
        // row r of a 128-byte-swizzled tile: 16-byte chunk c sits at chunk position c ^ (r & 7)
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const int off = r * 128 + ((c ^ (r & 7)) << 4);
          const uint4 gv = *reinterpret_cast<const uint4*>(sdO + off);
          const uint4 ov = *reinterpret_cast<const uint4*>(sO + off);
          const uint32_t* gw = reinterpret_cast<const uint32_t*>(&gv);
          const uint32_t* ow = reinterpret_cast<const uint32_t*>(&ov);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float2 a2 = Cvt<T>::unpack2(ow[i]), g2 = Cvt<T>::unpack2(gw[i]);
            dlt = fmaf(a2.x, g2.x, dlt);
            dlt = fmaf(a2.y, g2.y, dlt);
          }
        }
        if (grow < S) DELTA[(int64_t)bh * S + grow] = dlt;
      }
    } else {
      dlt = grow < S ? DELTA[(int64_t)bh * S + grow] : 0.f;
    }
    [[maybe_unused]] const uint64_t sc2 = f2_pack(scale2, scale2), nl2 = f2_pack(-lse2, -lse2), nd2 = f2_pack(-dlt, -dlt);
    for (int j = 0; ok && j < nkv; ++j) {
      if (!warp_wait(&ctl->sdp_full, j & 1, abort_flag)) { if (lane == 0) atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_MMA); ok = false; break; }
      fence_after_sync();
      uint32_t sv[2][32], pv[2][32], pk[32];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) { tmem_ld32(t_row + hf * 32, sv[hf]); tmem_ld32(t_row + kColDP + hf * 32, pv[hf]); }
      tmem_wait_ld();
      fence_before_sync();
      warp_arrive(&ctl->sdp_free);                       // both are in registers: the next tile's may come
      const int c0 = j * BT;
      const int lim = (CAUSAL && grow < S ? grow : S - 1) - c0;   // last visible key of this row within the tile
      // The masked and the unmasked form of a tile are separate code: as one body the compiler predicates the
      // mask's compare-and-select per element, and predicated-off instructions still take issue slots in the
      // tiles that need no mask (all but one or two per item).
      auto tile_body = [&](auto edge_c) {
        constexpr bool EDGE = decltype(edge_c)::value;
#pragma unroll
        for (int c = 0; c < BT; c += 2) {
          float d2[2];
          const uint32_t s0 = sv[c >> 5][c & 31], s1 = sv[c >> 5][(c & 31) + 1], g0 = pv[c >> 5][c & 31], g1 = pv[c >> 5][(c & 31) + 1];
          if constexpr (!DROPOUT) {
            pair_ds(s0, s1, g0, g1, sc2, nl2, nd2, [&](int e) { return !EDGE || c + e <= lim; }, d2);
          } else {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              float p = ex2(fmaf(__uint_as_float(e ? s1 : s0), scale2, -lse2));
              if constexpr (EDGE) p = c + e <= lim ? p : 0.f;
              float dp = __uint_as_float(e ? g1 : g0);
              dp = dropout_keep(seed_mix, grow, c0 + c + e, dropout_p) ? dp * inv_keep : 0.f;
              d2[e] = p * (dp - dlt);
            }
          }
          pk[c >> 1] = Cvt<T>::pack2(d2[0], d2[1]);
        }
      };
      if ((CAUSAL && c0 + BT - 1 > m0 + warp * 32) || c0 + BT > S) tile_body(std::true_type{}); else tile_body(std::false_type{});
      // dS_{j-1} must have been read; its MMAs were issued a tile ago
      if (j > 0 && !warp_wait(&ctl->dq_done, (j - 1) & 1, abort_flag)) { if (lane == 0) atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_MMA); ok = false; break; }
      fence_after_sync();
      tmem_st32(t_row + kColDS, pk);
      tmem_wait_st();
      fence_before_sync();
      warp_arrive(&ctl->ds_ready);
    }
    // epilogue: the four warps go through it together or not at all (its staging tile is shared)
    const int tg = (int)threadIdx.x;
    [[maybe_unused]] RopeQuad tab[kRopeTasks];
    if constexpr (ROPE) rope_prefetch_pass(tab, rt, m0, 0, tg, S);   // ahead of the wait for the last gradient MMAs
    if (ok && !warp_wait(&ctl->dq_done, (nkv - 1) & 1, abort_flag)) { if (lane == 0) atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_MMA); ok = false; }
    if (!quad_any(!ok)) {
      fence_after_sync();
      uint4 lo[4], hi[4];
      acc_to_16bit<T>(t_row + kColDQ, scale, lo);
      acc_to_16bit<T>(t_row + kColDQ + 32, scale, hi);
      T* item_out = dQ + (int64_t)b * dq_sb + (int64_t)h * dq_sh + (int64_t)m0 * dq_ss;
      if constexpr (ROPE) {
        rope_adjoint_store<T>(sQ, tg, r, lo, hi, item_out, dq_ss, m0, S, rt, tab);
      } else {
        staged_store<T>(sQ + warp * kWarpStageBytes, lane, lo, hi, item_out + (int64_t)(warp * 32) * dq_ss, dq_ss, S - m0 - warp * 32);
      }
    }
  }

  fence_before_sync();
  __syncthreads();
  if (warp == 5) tmem_dealloc(tmem_base, kTmemColsQ);
  if (threadIdx.x == 0 && ctl->fail_bits && status) atomicOr(status, ctl->fail_bits);
}

// ---------------------------------------------------------------------------
// dK / dV kernel
// A work item is one (batch*head, key tile of 128); key tile 0 meets the most query tiles under the
// causal mask, so items are numbered by key tile, ascending: heaviest first.
// Persistent: one CTA per SM walks a static list of items, dealt in boustrophedon order (ItemIter), which balances the CTAs' totals to
// within one item of the mean without a global counter.  Every role walks the same list, and all ring / buffer indices run on a
// tile counter that keeps counting across items, so the producer prefetches the next item's resident tiles (double-buffered) and
// first streamed tiles, and the S and dP issuers fill free score buffers with them, while the last tiles of the current item are
// still being worked on.  Only the gradient issuer pauses between items, until the accumulators have been read out of TMEM.
// Two compute groups of four warps take alternate query tiles, each in TMEM columns of its own.  A compute thread owns a key row: it
// takes the 64 + 64 values of its row into registers and hands both buffers back at once, so the group's next S^T and dP^T are there
// when it has written this tile's P^T and dS^T, into columns that the gradient MMAs of its previous tile have long read.
// Finished gradients leave through a warpgroup of its own: done by a compute group, the 6,500 clk between an item's last gradient
// MMA and its stores held up the tiles of the next item, 12 % of the kernel's time at S = 4096.
// What bounds it: at B8 H12 S4096 a CTA runs 730,000 clk, 2,130 for each of a group's 342 tiles.  1,900 of them are the group's loop,
// of which 1,330 are arithmetic (issue slots and the SFU, shared with the other group) and the rest synchronisation whose
// instructions queue behind the exponentials; 230 a tile, 3,800 an item, are the change of item, start-up and the end.  The SFU is
// at 48 % of its peak, the tensor pipe at 48 %, issue slots at 49 %.  Against three groups of eight warps over three score buffer
// pairs, P and dS packed over the scores, on one GPU (us): B8 H12 S4096 bf16 470 -> 450, B24 H12 S1363 fp16 222 -> 202, B64 H12
// S300 68.7 -> 61.5, B1 H16 S4096 85 -> 76.5, B4 H12 S201 8.9 -> 8.6, B1 H12 S67 6.8 -> 6.7, B1 H2 S32 6.0 -> 6.2.  The groups
// taking strict turns with their exponentials: 489 (turns of 1,000 clk each leave no more than they give).
// ---------------------------------------------------------------------------
struct CtlKV {
  uint64_t kv_full[2], kv_free[2], qdo_full[kStages], qdo_empty[kStages], sdp_full[kGroups], sdp_free[kGroups], pds_ready[kGroups],
      grad_done[kGroups], dkv_done, acc_free;
  uint32_t tmem_base;
  int abort;
  uint32_t fail_bits;
  // Per-query statistics of each streamed tile: -lse in log2 units, -delta (read as float4).  Written by the producer warp, read by the
  // compute warps; each hand-over goes along a chain of ordinary arrivals and waits: producer -> qdo_full -> S issuer -> sdp_full ->
  // compute warps, and back: compute warps -> pds_ready -> gradient issuer -> qdo_empty -> producer.
  alignas(16) float stat[kStages][2][BT];
};
constexpr size_t kCtlBytes = 4096;        // padded so that what follows stays 128-byte aligned
static_assert(sizeof(CtlKV) <= kCtlBytes, "control block");
constexpr uint32_t kGroupStageBytes = 4 * kWarpStageBytes;   // staging tile of the storing warps: 32 rows each, or a RoPE pass
static_assert(kGroupStageBytes >= kRopeStageBytes, "the RoPE adjoint's pass fits the staging tile");
constexpr size_t kSmemKV = 1024 + 4 * (size_t)kBigTile + (size_t)kStages * 2 * kSmallTile + kCtlBytes + kGroupStageBytes;
constexpr uint32_t kColG = 192;           // columns of a group: S^T at 0, dP^T at 64, packed P^T at 128, packed dS^T at 160
constexpr uint32_t kColV = kColG * kGroups, kColK = kColV + 64;

template <typename T, bool CAUSAL, bool DROPOUT, bool ROPE>
__global__ void __launch_bounds__(kThreadsKV, 1)
attn_bwd_dkv_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                    const float* __restrict__ LSE, const float* __restrict__ DELTA,
                    T* __restrict__ dK, T* __restrict__ dV,
                    int64_t dk_sb, int64_t dk_sh, int64_t dk_ss, int64_t dv_sb, int64_t dv_sh, int64_t dv_ss,
                    int S, int H, int BH, float scale, float scale2, float dropout_p, uint32_t seed, uint32_t* status,
                    const RopeTab rt) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sKVbig = base;                                 // [slot][K|V], 16 KB each; item n uses slot n & 1
  uint8_t* sQdO = base + 4 * kBigTile;                    // [stage][Q|dO], 8 KB each
  CtlKV* ctl = reinterpret_cast<CtlKV*>(sQdO + (size_t)kStages * 2 * kSmallTile);
  uint8_t* stage = reinterpret_cast<uint8_t*>(ctl) + kCtlBytes;   // the storing warps' staging tile
  volatile int* abort_flag = &ctl->abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_all = (S + BT - 1) / BT;
  const int n_items = BH * ((S + BR - 1) / BR);
  // item -> (batch*head, first key, first query tile, query tiles): key tile 0 is the heaviest under the causal mask
  auto decode = [&](int idx, int& bh, int& n0, int& i_begin, int& nq) {
    const int kt = idx / BH;
    bh = idx - kt * BH;
    n0 = kt * BR;
    i_begin = CAUSAL ? n0 / BT : 0;
    nq = n_all - i_begin;
  };

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(&ctl->kv_full[i], 1); mbar_init(&ctl->kv_free[i], 2); }
    // qdo_empty and sdp_full: the commits, and an arrival of the issuer itself that passes the statistics on (CtlKV::stat; a commit
    // stands for its MMAs alone).  B8 H12 S4096 448.9 -> 449.6 us, B24 H12 S1363 203.0 -> 201.6, shorter ones the same.
    for (int s = 0; s < kStages; ++s) { mbar_init(&ctl->qdo_full[s], 2); mbar_init(&ctl->qdo_empty[s], 2); }
    for (int g = 0; g < kGroups; ++g) {
      mbar_init(&ctl->sdp_full[g], 3); mbar_init(&ctl->sdp_free[g], kGroupWarps); mbar_init(&ctl->pds_ready[g], kGroupWarps);
      mbar_init(&ctl->grad_done[g], 1);
    }
    mbar_init(&ctl->dkv_done, 1);
    mbar_init(&ctl->acc_free, 4);
    ctl->abort = 0;
    ctl->fail_bits = 0;
    fence_mbar_init();
  }
  if (warp == kMmaWarp) { tmem_alloc(&ctl->tmem_base, kTmemCols); tmem_relinquish(); }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, ctl->tmem_base, 0);   // warp-uniform

  if (warp >= kStoreWarp) {
    // ------------------------------ gradients out -----------------------------
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsStore));
    const int sub = warp & 3, tg = (int)threadIdx.x & 127;
    const int r = tg;                                     // key row within the tile == TMEM lane
    const uint32_t t_row = tmem_base + ((uint32_t)(sub * 32) << 16);
    uint8_t* w_stage = stage + sub * kWarpStageBytes;
    ItemIter items(n_items);
    int idx;
    for (int n = 0; items.next(idx); ++n) {
      int bh, n0, i_begin, nq;
      decode(idx, bh, n0, i_begin, nq);
      const int b = bh / H, h = bh - b * H;
      // Fused RoPE adjoint on dK: the first pass's table values are fetched BEFORE the wait for the last gradient MMAs.
      [[maybe_unused]] RopeQuad tab[kRopeTasks];
      if constexpr (ROPE) rope_prefetch_pass(tab, rt, n0, 0, tg, S);
      const bool ok = warp_wait(&ctl->dkv_done, n & 1, abort_flag);
      if (!ok && lane == 0) atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_MMA);
      if (quad_any(!ok)) break;                    // the four warps leave together: their staging tile is shared
      fence_after_sync();
      // read and round everything first, hand the accumulators back, rotate dK (ROPE) and store afterwards
      T* v_item = dV + (int64_t)b * dv_sb + (int64_t)h * dv_sh + (int64_t)n0 * dv_ss;
      T* k_item = dK + (int64_t)b * dk_sb + (int64_t)h * dk_sh + (int64_t)n0 * dk_ss;
      uint4 vlo[4], vhi[4], klo[4], khi[4];
      acc_to_16bit<T>(t_row + kColV, 1.f, vlo);
      acc_to_16bit<T>(t_row + kColV + 32, 1.f, vhi);
      acc_to_16bit<T>(t_row + kColK, scale, klo);
      acc_to_16bit<T>(t_row + kColK + 32, scale, khi);
      fence_before_sync();
      warp_arrive(&ctl->acc_free);
      const int w0 = sub * 32;
      staged_store<T>(w_stage, lane, vlo, vhi, v_item + (int64_t)w0 * dv_ss, dv_ss, S - n0 - w0);
      if constexpr (ROPE) {
        quad_sync();                                 // the staging tile changes from a warp's to the group's
        rope_adjoint_store<T>(stage, tg, r, klo, khi, k_item, dk_ss, n0, S, rt, tab);
      } else {
        staged_store<T>(w_stage, lane, klo, khi, k_item + (int64_t)w0 * dk_ss, dk_ss, S - n0 - w0);
      }
    }
  } else if (warp >= kProducerWarp) {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));
  if (warp == kProducerWarp) {
    // The whole warp: one lane issues the copies, all of them bring the tiles' statistics (4-byte values at any offset, which TMA does
    // not take), fetched a tile ahead of the slot they go to.
    const bool leader = elect_one();
    if (leader) { tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmK); tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmdO); }
    ItemIter items(n_items);
    uint32_t t = 0;                                       // tiles issued so far, over all items
    int idx, idx_next, n_loaded = 0;                      // n_loaded: items whose K/V loads were issued
    auto load_item = [&](int item) -> bool {
      int bh, n0, i_begin, nq;
      decode(item, bh, n0, i_begin, nq);
      const int b = bh / H, h = bh - b * H, slot = n_loaded & 1;
      // the slot's previous K/V (two items ago) must have been read by the last S and dP MMAs of that item
      if (n_loaded >= 2 && !warp_wait(&ctl->kv_free[slot], ((n_loaded >> 1) - 1) & 1, abort_flag)) { if (leader) atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_MMA); return false; }
      if (leader) {
        uint8_t* big = sKVbig + (size_t)slot * 2 * kBigTile;
        mbar_expect_tx(&ctl->kv_full[slot], 2 * kBigTile);
        tma_load_4d(big, &tmK, &ctl->kv_full[slot], 0, n0, h, b);
        tma_load_4d(big + kBigTile, &tmV, &ctl->kv_full[slot], 0, n0, h, b);
      }
      ++n_loaded;
      return true;
    };
    bool have = items.next(idx);
    bool ok = have && load_item(idx);
    for (; ok && have; idx = idx_next) {
      int bh, n0, i_begin, nq;
      decode(idx, bh, n0, i_begin, nq);
      const int b = bh / H, h = bh - b * H;
      have = items.next(idx_next);
      float f_lse[BT / 32], f_dlt[BT / 32];
      auto fetch_stats = [&](int it) {
#pragma unroll
        for (int e = 0; e < BT / 32; ++e) {
          const int q = (i_begin + it) * BT + 32 * e + lane, qc = q < S ? q : S - 1;
          f_lse[e] = LSE[(int64_t)bh * S + qc];
          f_dlt[e] = DELTA[(int64_t)bh * S + qc];
        }
      };
      fetch_stats(0);
      for (int it = 0; it < nq; ++it, ++t) {
        const uint32_t s = t % kStages;
        if (t >= kStages && !warp_wait(&ctl->qdo_empty[s], ((t / kStages) - 1) & 1, abort_flag)) {
          if (leader) atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_MMA);
          ok = false;
          break;
        }
        if (leader) {
          uint8_t* dst = sQdO + (size_t)s * 2 * kSmallTile;
          mbar_expect_tx(&ctl->qdo_full[s], 2 * kSmallTile);
          tma_load_4d(dst, &tmQ, &ctl->qdo_full[s], 0, (i_begin + it) * BT, h, b);
          tma_load_4d(dst + kSmallTile, &tmdO, &ctl->qdo_full[s], 0, (i_begin + it) * BT, h, b);
        }
#pragma unroll
        for (int e = 0; e < BT / 32; ++e) {
          const bool in = (i_begin + it) * BT + 32 * e + lane < S;
          ctl->stat[s][0][32 * e + lane] = in ? -(f_lse[e] * kLog2e) : -INFINITY;
          ctl->stat[s][1][32 * e + lane] = in ? -f_dlt[e] : 0.f;
        }
        warp_arrive(&ctl->qdo_full[s]);
        if (it + 1 < nq) fetch_stats(it + 1);
        // the next item's resident tiles are requested behind the third tile of this one: the previous item is done with
        // their slot by then
        if (have && it == (nq > 3 ? 2 : nq - 1) && !load_item(idx_next)) { ok = false; ++t; break; }
      }
    }
    if (*abort_flag && leader) {   // let our own copies land before the CTA's shared memory goes away
      for (int m = n_loaded > 2 ? n_loaded - 2 : 0; m < n_loaded; ++m) {
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try(&ctl->kv_full[m & 1], (m >> 1) & 1))
          if (globaltimer_ns() - t0 > kWaitLimitNs) break;
      }
      for (uint32_t u = t > (uint32_t)kStages ? t - kStages : 0; u < t; ++u) {
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try(&ctl->qdo_full[u % kStages], (u / kStages) & 1))
          if (globaltimer_ns() - t0 > kWaitLimitNs) break;
      }
    }
  } else if (warp == kMmaWarp || warp == kMma2Warp) {
    if (elect_one()) {                                     // score MMAs: S^T = K Q_i^T (first issuer), dP^T = V dO_i^T (second)
      const bool second = warp == kMma2Warp;
      constexpr uint32_t idesc_s = make_idesc(Fmt<T>::v, BR, BT, 0);   // 128 keys x 64 queries
      ItemIter items(n_items);
      uint32_t t = 0;
      int n = 0, idx;
      bool ok = true;
      for (; ok && items.next(idx); ++n) {
        int bh, n0, i_begin, nq;
        decode(idx, bh, n0, i_begin, nq);
        const int slot = n & 1;
        if (!mbar_wait(&ctl->kv_full[slot], (n >> 1) & 1, abort_flag)) { atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_LOAD); break; }
        const uint64_t da = make_sdesc_sw128(smem_u32(sKVbig + (size_t)slot * 2 * kBigTile + (second ? kBigTile : 0)));
        for (int it = 0; it < nq; ++it, ++t) {
          const uint32_t s = t % kStages, g = t % kGroups;
          // the group has the values of its previous tile in registers
          if (t >= kGroups && !mbar_wait(&ctl->sdp_free[g], ((t / kGroups) - 1) & 1, abort_flag)) { atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_SOFTMAX); ok = false; break; }
          if (!mbar_wait(&ctl->qdo_full[s], (t / kStages) & 1, abort_flag)) { atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_LOAD); ok = false; break; }
          if (!second) mbar_arrive(&ctl->sdp_full[g]);    // passes the producer's statistics on to the group
          fence_after_sync();
          const uint64_t db = make_sdesc_sw128(smem_u32(sQdO + (size_t)s * 2 * kSmallTile + (second ? kSmallTile : 0)));
          const uint32_t t_dst = tmem_base + kColG * g + (second ? 64 : 0);
#pragma unroll
          for (int kk = 0; kk < HD / 16; ++kk) mma_ss(t_dst, da + (uint64_t)(kk * 2), db + (uint64_t)(kk * 2), idesc_s, kk > 0);
          mma_commit(&ctl->sdp_full[g]);
        }
        mma_commit(&ctl->kv_free[slot]);                  // arrives once this thread's MMAs of the item have read K (V)
      }
    }
  } else if (warp == kGradWarp) {
    if (elect_one()) {                                     // gradient MMAs: dV += P^T dO_i, dK += dS^T Q_i
      constexpr uint32_t idesc_a = make_idesc(Fmt<T>::v, BR, HD, 1);   // B = dO / Q tile read MN-major
      ItemIter items(n_items);
      uint32_t t = 0;
      int n = 0, idx;
      bool ok = true;
      for (; ok && items.next(idx); ++n) {
        int bh, n0, i_begin, nq;
        decode(idx, bh, n0, i_begin, nq);
        // the accumulators still hold the previous item's dK/dV until its epilogue has read them
        if (n >= 1 && !mbar_wait(&ctl->acc_free, (n - 1) & 1, abort_flag)) { atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_SOFTMAX); break; }
        fence_after_sync();
        for (int it = 0; it < nq; ++it, ++t) {
          const uint32_t s = t % kStages, g = t % kGroups;
          if (!mbar_wait(&ctl->pds_ready[g], (t / kGroups) & 1, abort_flag)) { atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_SOFTMAX); ok = false; break; }
          mbar_arrive(&ctl->qdo_empty[s]);                // the group has read the slot's statistics
          fence_after_sync();
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            // dV reads P^T against the dO tile; dK reads dS^T against the Q tile
            const bool sec = w == 1;
            const uint64_t db = make_sdesc_sw128(smem_u32(sQdO + (size_t)s * 2 * kSmallTile + (sec ? 0 : kSmallTile)));
            const uint32_t t_acc = tmem_base + (sec ? kColK : kColV), t_a = tmem_base + kColG * g + (sec ? 160 : 128);
#pragma unroll
            for (int kk = 0; kk < BT / 16; ++kk)
              mma_ts(t_acc, t_a + (uint32_t)(kk * 8), db + (uint64_t)(kk * (2048 >> 4)), idesc_a, (it > 0 || kk > 0) ? 1u : 0u);
          }
          mma_commit(&ctl->grad_done[g]);
          mma_commit(&ctl->qdo_empty[s]);
        }
        if (ok) mma_commit(&ctl->dkv_done);
      }
    }
  }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsCompute));
    const int g = warp / kGroupWarps;
    const int sub = warp & 3;                             // TMEM sub-partition = scheduler
    const int r = sub * 32 + lane;                        // key row within the tile == TMEM lane
    const uint32_t t_grp = tmem_base + ((uint32_t)(sub * 32) << 16) + kColG * g;
    [[maybe_unused]] const uint64_t sc2 = f2_pack(scale2, scale2);
    const float inv_keep = DROPOUT ? 1.f / (1.f - dropout_p) : 1.f;
    ItemIter items(n_items);
    uint32_t t0 = 0;                                      // tile counter at the start of the item
    uint32_t mine = 0;                                    // tiles this group has worked on: the phase of its barriers
    int idx;
    bool ok = true;
    while (ok && items.next(idx)) {
      int bh, n0, i_begin, nq;
      decode(idx, bh, n0, i_begin, nq);
      const int kc = n0 + r;                              // this thread's key
      const uint32_t seed_mix = (seed * 0x9E3779B1u) ^ (((uint32_t)bh + 1u) * 0x27D4EB2Fu);
      // tile t belongs to group t % kGroups, counted over all items
      for (int it = (int)((g + kGroups - t0 % kGroups) % kGroups); it < nq; it += kGroups, ++mine) {
        const int i0 = (i_begin + it) * BT;
        const float* w_lse = ctl->stat[(t0 + (uint32_t)it) % kStages][0];
        const float* w_dlt = w_lse + BT;
        if (!warp_wait(&ctl->sdp_full[g], mine & 1, abort_flag)) { if (lane == 0) atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_MMA); ok = false; break; }
        fence_after_sync();
        // The statistics are read two chunks of queries ahead of their use: a shared-memory load queues behind the
        // exponentials that were issued before it.
        constexpr int kStat = 4;
        float st[3][2 * kStat];
        auto load_stats = [&](int cc) {
#pragma unroll
          for (int v = 0; v < kStat; v += 4) {
            lds_f4(w_lse + cc * kStat + v, st[cc % 3] + v);
            lds_f4(w_dlt + cc * kStat + v, st[cc % 3] + kStat + v);
          }
        };
        uint32_t sv[2][32], pv[2][32], pp[16], pd[16];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) { tmem_ld32(t_grp + hf * 32, sv[hf]); tmem_ld32(t_grp + 64 + hf * 32, pv[hf]); }
        load_stats(0);
        load_stats(1);
        tmem_wait_ld();
        fence_before_sync();
        warp_arrive(&ctl->sdp_free[g]);                   // both are in registers: the group's next tile may come
        const int first = kc - i0;                        // the first query of the tile that sees this key
        auto tile_body = [&](auto edge_c) {                // masked / unmasked tiles as separate code (see the dQ kernel)
          constexpr bool EDGE = decltype(edge_c)::value;
#pragma unroll
          for (int cc = 0; cc < BT / kStat; ++cc) {
            if (cc + 2 < BT / kStat) load_stats(cc + 2);
            const float* l8 = st[cc % 3];
            const float* d8 = st[cc % 3] + kStat;
#pragma unroll
            for (int i = 0; i < kStat; i += 2) {
              const int c = cc * kStat + i;
              float p2[2], d2[2];
              const uint32_t s0 = sv[c >> 5][c & 31], s1 = sv[c >> 5][(c & 31) + 1], g0 = pv[c >> 5][c & 31], g1 = pv[c >> 5][(c & 31) + 1];
              if constexpr (!DROPOUT) {
                pair_ds(s0, s1, g0, g1, sc2, f2_pack(l8[i], l8[i + 1]), f2_pack(d8[i], d8[i + 1]),
                        [&](int e) { return !EDGE || c + e >= first; }, d2, p2);
              } else {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  float p = ex2(fmaf(__uint_as_float(e ? s1 : s0), scale2, l8[i + e]));
                  if constexpr (EDGE) p = c + e >= first ? p : 0.f;
                  float dp = __uint_as_float(e ? g1 : g0);
                  const bool keep = dropout_keep(seed_mix, i0 + c + e, kc, dropout_p);
                  p2[e] = keep ? p * inv_keep : 0.f;
                  dp = keep ? dp * inv_keep : 0.f;
                  d2[e] = p * (dp + d8[i + e]);
                }
              }
              pp[(c >> 1) & 15] = Cvt<T>::pack2(p2[0], p2[1]);
              pd[(c >> 1) & 15] = Cvt<T>::pack2(d2[0], d2[1]);
            }
            if (cc == BT / kStat / 2 - 1) {
              // the group's previous P^T and dS^T must have been read; their MMAs were issued a tile ago
              if (mine > 0 && !warp_wait(&ctl->grad_done[g], (mine - 1) & 1, abort_flag)) { if (lane == 0) atomicOr(&ctl->fail_bits, (uint32_t)ULM_STATUS_TIMEOUT_MMA); ok = false; }
              fence_after_sync();
              st16(t_grp + 128, pp);
              st16(t_grp + 160, pd);
            }
          }
          st16(t_grp + 144, pp);
          st16(t_grp + 176, pd);
        };
        if (CAUSAL && i0 < n0 + sub * 32 + 31) tile_body(std::true_type{}); else tile_body(std::false_type{});   // some query of the tile precedes some key of the warp
        if (!ok) break;
        tmem_wait_st();
        fence_before_sync();
        warp_arrive(&ctl->pds_ready[g]);
      }
      t0 += (uint32_t)nq;
    }
  }

  fence_before_sync();
  __syncthreads();
  if (warp == kMmaWarp) tmem_dealloc(tmem_base, kTmemCols);
  if (threadIdx.x == 0 && ctl->fail_bits && status) atomicOr(status, ctl->fail_bits);
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
struct Maps { CUtensorMap q128, q64, k128, k64, v128, v64, do128, do64, o128; };

// SMs of the current device (the persistent kernels launch one CTA on each)
int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return kNumSMs;
  return n;
}

template <typename T, bool CAUSAL, bool DROPOUT, bool ROPE>
int launch_bwd(const ulm_attn_bwd_args* a, int device, const Maps& m) {
  cudaStream_t st = (cudaStream_t)a->stream;
  const unsigned BH = (unsigned)(a->B * a->H);
  const unsigned nt = (unsigned)((a->S + BR - 1) / BR);
  const float scale2 = a->softmax_scale * kLog2e;
  RopeTab rt{};
  if (ROPE) rt = RopeTab{a->cos_tab, a->sin_tab, a->cos_stride, a->sin_stride};
  int rc = ULM_OK;
  const bool fuse_delta = (a->mode & 3) == 3;            // delta wanted and the dQ kernel runs: it computes delta itself
  if ((a->mode & 1) && !fuse_delta) {
    dim3 g((unsigned)((a->S + 31) / 32), BH);
    attn_delta_kernel<T><<<g, 256, 0, st>>>((const T*)a->o, (const T*)a->d_o, a->delta, a->o_sb, a->o_sh, a->o_ss,
                                            a->do_sb, a->do_sh, a->do_ss, a->S, a->H);
    if ((rc = check_launch("ulm_attn_bwd(delta)"))) return rc;
  }
  const unsigned items = BH * nt;
  const unsigned grid = items < (unsigned)sm_count() ? items : (unsigned)sm_count();
  if (a->mode & 2) {
    auto go = [&](auto kern, std::atomic<bool>* attr) -> int {
      if (int r = ensure_smem_attr(kern, kSmemQ, device, attr, "ulm_attn_bwd(dq)")) return r;
      kern<<<dim3(BH, nt), kThreadsQ, kSmemQ, st>>>(m.q128, m.k64, m.v64, m.do128, m.o128, a->lse, a->delta, (T*)a->dq,
                                                          a->dq_sb, a->dq_sh, a->dq_ss, a->S, a->H, a->softmax_scale, scale2,
                                                          a->dropout_p, a->seed, a->status_dev, rt);
      return check_launch("ulm_attn_bwd(dq)");
    };
    static std::atomic<bool> attr_fused[kMaxDevices], attr_plain[kMaxDevices];
    rc = fuse_delta ? go(attn_bwd_dq_kernel<T, CAUSAL, DROPOUT, true, ROPE>, attr_fused)
                    : go(attn_bwd_dq_kernel<T, CAUSAL, DROPOUT, false, ROPE>, attr_plain);
    if (rc) return rc;
  }
  if (a->mode & 4) {
    auto kern = attn_bwd_dkv_kernel<T, CAUSAL, DROPOUT, ROPE>;
    static std::atomic<bool> attr[kMaxDevices];
    const size_t smem = kSmemKV;
    if ((rc = ensure_smem_attr(kern, smem, device, attr, "ulm_attn_bwd(dkv)"))) return rc;
    kern<<<grid, kThreadsKV, smem, st>>>(m.q64, m.k128, m.v128, m.do64, a->lse, a->delta, (T*)a->dk, (T*)a->dv,
                                          a->dk_sb, a->dk_sh, a->dk_ss, a->dv_sb, a->dv_sh, a->dv_ss,
                                          a->S, a->H, (int)BH, a->softmax_scale, scale2, a->dropout_p, a->seed, a->status_dev, rt);
    if ((rc = check_launch("ulm_attn_bwd(dkv)"))) return rc;
  }
  return rc;
}

template <typename T, bool ROPE>
int dispatch_bwd(const ulm_attn_bwd_args* a, int device, const Maps& m) {
  const bool drop = a->dropout_p > 0.f;
  if (a->causal) return drop ? launch_bwd<T, true, true, ROPE>(a, device, m) : launch_bwd<T, true, false, ROPE>(a, device, m);
  return drop ? launch_bwd<T, false, true, ROPE>(a, device, m) : launch_bwd<T, false, false, ROPE>(a, device, m);
}

bool ok_out(const void* p, int64_t sb, int64_t sh, int64_t ss) {
  return p && !(reinterpret_cast<uintptr_t>(p) & 15) && sb % 8 == 0 && sh % 8 == 0 && ss % 8 == 0;
}

}  // namespace
}  // namespace ulm

extern "C" int ulm_attn_bwd(const ulm_attn_bwd_args* a) {
  using namespace ulm;
  if (!a) return fail(ULM_ERR_ARG, "ulm_attn_bwd: null args");
  if (a->dtype != ULM_F16 && a->dtype != ULM_BF16) return fail(ULM_ERR_ARG, "ulm_attn_bwd: dtype must be f16 or bf16");
  if (a->B < 0 || a->H < 0 || a->S < 0) return fail(ULM_ERR_ARG, "ulm_attn_bwd: negative size");
  if (a->B == 0 || a->H == 0 || a->S == 0 || (a->mode & 7) == 0) return ULM_OK;
  if (!a->q || !a->k || !a->v || !a->d_o || !a->lse || !a->delta) return fail(ULM_ERR_ARG, "ulm_attn_bwd: null tensor");
  if (!(a->softmax_scale > 0.f)) return fail(ULM_ERR_ARG, "ulm_attn_bwd: softmax_scale must be positive");
  if (a->dropout_p < 0.f || a->dropout_p >= 1.f) return fail(ULM_ERR_ARG, "ulm_attn_bwd: dropout_p must be in [0,1)");
  if ((a->mode & 1) && !ok_out(a->o, a->o_sb, a->o_sh, a->o_ss)) return fail(ULM_ERR_ARG, "ulm_attn_bwd: o must be 16-byte aligned, strides multiples of 8");
  if ((a->mode & 2) && !ok_out(a->dq, a->dq_sb, a->dq_sh, a->dq_ss)) return fail(ULM_ERR_ARG, "ulm_attn_bwd: dq must be 16-byte aligned, strides multiples of 8");
  if ((a->mode & 4) && (!ok_out(a->dk, a->dk_sb, a->dk_sh, a->dk_ss) || !ok_out(a->dv, a->dv_sb, a->dv_sh, a->dv_ss)))
    return fail(ULM_ERR_ARG, "ulm_attn_bwd: dk/dv must be 16-byte aligned, strides multiples of 8");
  if ((int64_t)a->B * a->H > 0x7fffffffLL || (a->S + 31) / 32 > 65535 * 4) return fail(ULM_ERR_TOO_LARGE, "ulm_attn_bwd: grid too large");
  const bool rope = a->cos_tab || a->sin_tab;
  if (rope) {
    if (!a->cos_tab || !a->sin_tab) return fail(ULM_ERR_ARG, "ulm_attn_bwd: cos_tab and sin_tab must be given together");
    if ((reinterpret_cast<uintptr_t>(a->cos_tab) & 15) || (reinterpret_cast<uintptr_t>(a->sin_tab) & 15) || a->cos_stride % 4 || a->sin_stride % 4 ||
        a->cos_stride < 64 || a->sin_stride < 64)
      return fail(ULM_ERR_ARG, "ulm_attn_bwd: RoPE tables must be 16-byte aligned with row strides that are multiples of 4 floats, at least 64");
  }
  tc::DeviceScope dev(a->q, "ulm_attn_bwd");
  if (dev.rc) return dev.rc;
  Maps m{};
  int rc;
#define ULM_MAP(dst, ptr, sb, sh, ss, rows, what) \
  if ((rc = tc::encode_bhsd_map(&m.dst, a->ptr, a->dtype, a->B, a->H, a->S, a->sb, a->sh, a->ss, rows, what))) return rc
  if (a->mode & 2) {
    ULM_MAP(q128, q, q_sb, q_sh, q_ss, BR, "ulm_attn_bwd(q)");
    ULM_MAP(k64, k, k_sb, k_sh, k_ss, BT, "ulm_attn_bwd(k)");
    ULM_MAP(v64, v, v_sb, v_sh, v_ss, BT, "ulm_attn_bwd(v)");
    ULM_MAP(do128, d_o, do_sb, do_sh, do_ss, BR, "ulm_attn_bwd(do)");
  }
  if (a->mode & 4) {
    ULM_MAP(q64, q, q_sb, q_sh, q_ss, BT, "ulm_attn_bwd(q)");
    ULM_MAP(k128, k, k_sb, k_sh, k_ss, BR, "ulm_attn_bwd(k)");
    ULM_MAP(v128, v, v_sb, v_sh, v_ss, BR, "ulm_attn_bwd(v)");
    ULM_MAP(do64, d_o, do_sb, do_sh, do_ss, BT, "ulm_attn_bwd(do)");
  }
  if ((a->mode & 3) == 3) ULM_MAP(o128, o, o_sb, o_sh, o_ss, BR, "ulm_attn_bwd(o)");   // the dQ kernel computes delta itself
#undef ULM_MAP
  if (a->dtype == ULM_F16) return rope ? dispatch_bwd<__half, true>(a, dev.device, m) : dispatch_bwd<__half, false>(a, dev.device, m);
  return rope ? dispatch_bwd<__nv_bfloat16, true>(a, dev.device, m) : dispatch_bwd<__nv_bfloat16, false>(a, dev.device, m);
}
