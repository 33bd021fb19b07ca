// gnm_tensor.cu — the tcgen05 tensor engine (many score columns) and the
// re-unpacking backward kernel dW = G^T dS, each on BF16 limbs (kind::f16)
// and on 8-bit integer limbs (kind::i8):
//   gnm_tc_accumulate / gnm_t8_accumulate  wide: scores as M, one SM per tile
//   gnm_t8_pairs                           wide, 8-bit, SM pairs (cta_group::2),
//                                          one persistent launch per call
//   gnm_t8_narrow                          8-bit, people as M: the default but for
//                                          large limbs and some score counts
//                                          (prefers_people)
//   gnm_tc_narrow                          the same on BF16 limbs (<= 64 scores)
//   gnm_tc_backward                        dW = G^T dS, dC on CUDA cores
//   gnm_t8_backward                        dW and dC on the tensor cores (default)
// The BF16 forms come first below; each 8-bit form states what it changes.
//
// Scoring as a GEMM (the reference does this with three cuBLAS SGEMMs per
// score tile, score/cuda_backend.rs:2196-2233):
//   sum[p,k] = baseline[k] + sum_v W'[k,v] d(p,v) - sum_v C[k,v] m(p,v)
//   miss[p,k] = sum_v member[k,v] m(p,v)
// with d the allele-2 dosage (missing -> 0), m the missing indicator.
//
// Precision (the "hi/mid/lo" split): every weight-like value x of score k is
// written as hi + mid + lo (+ lo2 for dosage weights), each an integer multiple
// of a power-of-two quantum (q, q/2^8, q/2^16, q/2^24 with 2^E = 256 q >= max |x|
// of the score), |integer| <= 256, so every limb is exact in BF16.  Products with
// d in {0,1,2} and m in {0,1} are exact, every partial sum of one limb is an
// integer multiple of its quantum, and below 32768 variants its magnitude stays
// under 2^24 quanta: the FP32 tensor-memory accumulation of each limb is EXACT.
// Accumulators are flushed to FP64 every 16384 variants (the cross-block
// reduction is the only FP64 arithmetic).  The only error left is the limb
// residual: below 2^-33 of the score's largest weight for dosage weights (four
// limbs; with three it was 2^-25, and ~10^5 such residuals per sum reached
// 1e-6 of the score) and 2^-25 for missing corrections (three limbs; they touch
// only the ~1% missing calls).
//
// Kernel shape (one CTA per SM): M = 128 score rows (TMEM lanes), N = 256
// people (TMEM columns), K = 64 variants per stage, two limb planes per pass
// (2 x 256 FP32 accumulator columns fill the 512 TMEM columns), three stages
// of 68 KB in shared memory.  With 256 people per CTA every weight byte
// staged from L2 feeds twice the MMA work of a 128-person tile; the four
// passes (dosage limbs 0-1, dosage limbs 2-3, correction limbs 0-1,
// correction limb 2 + member count) each re-expand the genotypes, which is
// cheap CUDA-core work on separate warps.  Warp 0 issues TMA (weight limb
// planes, 3D map, 128-byte swizzle; packed rows, 2D map), warp 1 owns TMEM
// and issues tcgen05.mma, warps 2-5 expand packed 2-bit genotypes into the
// BF16 K-major operand in shared memory and drain TMEM at block ends.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "gnm_device.cuh"
#include "gnm_plan.h"
#include "gnm_tcgen05.cuh"
#include "gnm_tensor.h"

namespace gnm {

constexpr uint32_t kTcM = 128;        // score rows per tile
constexpr uint32_t kTcN = 256;        // people per tile
constexpr uint32_t kTcK = 64;         // variants per stage
constexpr uint32_t kTcFlush = 256;    // stages per exact FP32 block (16384 variants)
constexpr uint32_t kTcThreads = 192;  // 6 warps
constexpr int kTcPlanes = 2;          // limb planes per pass (2 x 256 TMEM columns)
constexpr int kTcStages = 3;          // pipeline stages (68 KB each)
constexpr uint64_t kNarrowMaxScores = 64;   // up to 4 narrow score tiles

struct TensorPlan {
  uint64_t K_pad = 0, V_pad = 0, P_pad = 0;
  uint32_t ptiles = 0, stiles = 0;
  __nv_bfloat16* d_planes_dos = nullptr;  // [4][K_pad][V_pad] W' limbs
  __nv_bfloat16* d_planes_mis = nullptr;  // [4][K_pad][V_pad] -corr limbs, member
  double* d_part_sum = nullptr;           // wide kernels: [K_pad][P_pad]
  uint32_t* d_part_cnt = nullptr;
  double* d_slot_sum = nullptr;           // people as M: [slots][K16][P_nar]; up to 64 scores
  uint32_t* d_slot_cnt = nullptr;         //   the same memory as d_part_sum / d_part_cnt
  bool slots_used = false;                // over 64 scores: slots written since the last reset
  uint32_t nsplits = 1;                   // narrow BF16: variant splits (grid z)
  uint32_t nscores = 1;                   // narrow 8-bit: 16-score groups per CTA (narrow_scores)
  uint64_t P_nar = 0;                     // narrow: people rounded up to 512
  uint64_t nslot = 0;                     // narrow: elements per slot (K16 * P_nar)
  uint32_t nalloc = 0;                    // narrow: slots allocated
  uint32_t nslots8 = 0;                   // narrow 8-bit: the most slots a call uses
  uint32_t sms = 1;
  uint32_t* d_state = nullptr;            // narrow: slot state (slots_written)
  bool wide_clear = false;                // wide partials cleared since the last reset
  CUtensorMap map_dos, map_mis;
  int8_t* d_planes8 = nullptr;            // [9][K_pad][V_pad8] 8-bit limbs (dosage, -corr, member)
  double* d_quanta8 = nullptr;            // [9][K_pad] quantum of each 8-bit plane
  uint64_t V_pad8 = 0;
  CUtensorMap map8_2, map8_1;             // boxes of two planes / one plane
  bool i8 = false;                        // wide GEMM on 8-bit limbs (gnm_t8_accumulate)
  bool pair = false;                      // ... over SM pairs (gnm_t8_pairs)
  double* d_part_pass = nullptr;          // SM pairs, passes 1-3: [3][K_pad][P_pad]
  bool pass_valid = false;                // d_part_pass written since the last reset
  bool narrow = false;                    // up to 64 scores: people as M (8-bit or BF16 limbs)
  bool can_narrow = false;                // K <= 64: either kernel can run the plan
  bool people = false;                    // the default shape runs people as M
  bool pinned_people = false;             // over 64 scores: a shape that names people as M
  uint32_t exact = 0;                     // kShapeExact of the shape
  CUtensorMap nmap_dos, nmap_mis;         // narrow boxes: 16 scores x 4 planes
  CUtensorMap nmap8_dos, nmap8_mis;       // 8-bit boxes: 128 variants x 16 nscores x 4 / 5 planes
};

struct TcArgs {
  uint64_t num_rows;       // rows of this block
  int32_t a_x0;            // absolute variant index of block row 0 (multiple of 64)
  double* part_sum;
  uint32_t* part_cnt;
  uint64_t P_pad;
  uint32_t* err;
  uint32_t raster;         // 0: blockIdx.x = people tile, 1: blockIdx.x = score tile
  int32_t z0;              // first limb plane of this pass (TMA z coordinate)
};

template <int NP, int ST>
struct TcSmem {
  static constexpr uint32_t kPlane = kTcM * kTcK * 2;   // 16 KB
  static constexpr uint32_t kAStage = NP * kPlane;
  static constexpr uint32_t kB = kTcN * kTcK * 2;       // 32 KB
  static constexpr uint32_t kPk = kTcK * (kTcN / 4);    // 4 KB
  static constexpr uint32_t kAOff = 0;
  static constexpr uint32_t kBOff = kAOff + ST * kAStage;
  static constexpr uint32_t kPkOff = kBOff + ST * kB;
  static constexpr uint32_t kBarOff = kPkOff + ST * kPk;
  static constexpr uint32_t kHolder = kBarOff + 8 * (3 * ST + 2);
  static constexpr uint32_t kTotal = kHolder + 16 + 1024;  // + alignment slack
};

// code -> BF16 byte tables for __byte_perm (pool bytes 0-3: low bytes by
// code, 4-7: high bytes by code).  Dosage: 00->0, 01(missing)->0, 10->1, 11->2.
// Missing indicator: 01 -> 1, else 0.
constexpr uint32_t kDosLo = 0x00800000u, kDosHi = 0x403F0000u;
constexpr uint32_t kMisLo = 0x00008000u, kMisHi = 0x00003F00u;

__device__ __forceinline__ uint32_t bf16_pair(uint32_t y16, uint32_t lo, uint32_t hi) {
  return __byte_perm(lo, hi, y16 * 0x11u + 0x4040u);
}

// MISSING: the B operand is the missing indicator (else the dosage).
// COUNT_LAST: the pass's last plane is the member plane; its products are the
// missing counts (else every plane is a limb of the pass's sum).
template <int NP, int ST, bool MISSING, bool COUNT_LAST>
__global__ void __launch_bounds__(kTcThreads, 1)
    gnm_tc_accumulate(const __grid_constant__ CUtensorMap amap,
                      const __grid_constant__ CUtensorMap pmap, TcArgs a) {
  using L = TcSmem<NP, ST>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sb = smem_u32(smem);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ptile = a.raster ? blockIdx.y : blockIdx.x;
  const uint32_t stile = a.raster ? blockIdx.x : blockIdx.y;
  const uint32_t nit = uint32_t((a.num_rows + kTcK - 1) / kTcK);
  auto full = [&](uint32_t s) { return sb + L::kBarOff + 8 * s; };
  auto bready = [&](uint32_t s) { return sb + L::kBarOff + 8 * (ST + s); };
  auto empty = [&](uint32_t s) { return sb + L::kBarOff + 8 * (2 * ST + s); };
  const uint32_t accfull = sb + L::kBarOff + 8 * (3 * ST);
  const uint32_t accempty = sb + L::kBarOff + 8 * (3 * ST + 1);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L::kHolder + 8);
  const uint32_t abort_addr = sb + L::kHolder + 8;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < ST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(bready(s), 128);
      mbar_init(empty(s), 1);
    }
    mbar_init(accfull, 1);
    mbar_init(accempty, 128);
    *abort_flag = 0u;
    fence_mbar_init();
    prefetch_tmap(&amap);
    prefetch_tmap(&pmap);
  }
  if (warp == 1) {
    tmem_alloc(sb + L::kHolder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + L::kHolder);

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      for (uint32_t it = 0; it < nit; ++it) {
        const uint32_t s = it % ST, ph = (it / ST) & 1u;
        if (!mbar_wait_bounded(empty(s), ph ^ 1u)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        if (lds_volatile_u32(abort_addr)) break;
        mbar_arrive_expect_tx(full(s), L::kAStage + L::kPk);
        tma_load_3d(sb + L::kAOff + s * L::kAStage, &amap, a.a_x0 + int32_t(it * kTcK),
                    int32_t(stile * kTcM), a.z0, full(s));
        tma_load_2d(sb + L::kPkOff + s * L::kPk, &pmap, int32_t(ptile * (kTcN / 4)),
                    int32_t(it * kTcK), full(s));
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_bf16_f32(kTcM, kTcN);
      uint32_t blk = 0;
      for (uint32_t it = 0; it < nit; ++it) {
        const uint32_t s = it % ST, ph = (it / ST) & 1u;
        const bool first = (it % kTcFlush) == 0;
        if (first && it > 0) {
          if (!mbar_wait_bounded(accempty, (blk - 1) & 1u)) {
            *abort_flag = 1u;
            atomicOr(a.err, kErrMmaTimeout);
            break;
          }
        }
        if (!mbar_wait_bounded(bready(s), ph)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        if (lds_volatile_u32(abort_addr)) break;
        tc_fence_after();
        const uint32_t a0 = sb + L::kAOff + s * L::kAStage;
        const uint32_t b0 = sb + L::kBOff + s * L::kB;
#pragma unroll
        for (uint32_t kk = 0; kk < kTcK / 16; ++kk) {
          const uint64_t bdesc = desc_kmajor_sw128(b0 + kk * 32);
#pragma unroll
          for (uint32_t j = 0; j < NP; ++j) {
            const uint64_t adesc = desc_kmajor_sw128(a0 + j * L::kPlane + kk * 32);
            tc_mma_f16(tmem + j * kTcN, adesc, bdesc, idesc, (first && kk == 0) ? 0u : 1u);
          }
        }
        tc_commit(empty(s));
        if ((it % kTcFlush) == kTcFlush - 1 || it == nit - 1) {
          tc_commit(accfull);
          ++blk;
        }
      }
    }
  } else {
    // ---------------- genotype expansion + epilogue (warps 2-5) ----------------
    const uint32_t pt = threadIdx.x - 64;      // 0..127
    const uint32_t col = pt & 31;              // byte column: people 4col..4col+3
    const uint32_t vg = pt >> 5;               // variant group: rows 16vg..16vg+15
    const uint32_t quad = warp & 3;            // TMEM lane quadrant of this warp
    uint32_t blk = 0;
    for (uint32_t it = 0; it < nit; ++it) {
      const uint32_t s = it % ST, ph = (it / ST) & 1u;
      if (!mbar_wait_bounded(full(s), ph)) {
        *abort_flag = 1u;
        atomicOr(a.err, kErrTmaTimeout);
        break;
      }
      if (lds_volatile_u32(abort_addr)) break;
      // explicit shared-space accesses: the realigned base is a generic pointer
      const uint32_t pk = sb + L::kPkOff + s * L::kPk;
      const uint32_t bt = sb + L::kBOff + s * L::kB;
#pragma unroll
      for (uint32_t h = 0; h < kTcN / 128; ++h) {
        const uint32_t bc = 32 * h + col;   // byte column: people 4bc..4bc+3
#pragma unroll
        for (uint32_t cc = 0; cc < 2; ++cc) {
          const uint32_t r0 = 16 * vg + 8 * cc;
          uint32_t xl = 0, xh = 0;
#pragma unroll
          for (uint32_t i = 0; i < 4; ++i) {
            xl |= lds_u8(pk + (r0 + i) * (kTcN / 4) + bc) << (8 * i);
            xh |= lds_u8(pk + (r0 + 4 + i) * (kTcN / 4) + bc) << (8 * i);
          }
          const uint32_t c = 2 * vg + cc;  // 16-byte chunk (8 variants) index
#pragma unroll
          for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t yl = (xl >> (2 * q)) & 0x03030303u;
            const uint32_t yh = (xh >> (2 * q)) & 0x03030303u;
            const uint32_t lo = MISSING ? kMisLo : kDosLo, hi = MISSING ? kMisHi : kDosHi;
            uint4 v;
            v.x = bf16_pair(yl & 0xFFFFu, lo, hi);
            v.y = bf16_pair(yl >> 16, lo, hi);
            v.z = bf16_pair(yh & 0xFFFFu, lo, hi);
            v.w = bf16_pair(yh >> 16, lo, hi);
            // operand row of person 128h + 4col + q (conflict-free 16-byte stores)
            const uint32_t n = 128 * h + 32 * q + col;
            sts_u128(bt + (n >> 3) * 1024 + (n & 7) * 128 + ((c ^ (n & 7)) << 4), v);
          }
        }
      }
      fence_proxy_async_smem();
      mbar_arrive(bready(s));

      if ((it % kTcFlush) == kTcFlush - 1 || it == nit - 1) {
        if (!mbar_wait_bounded(accfull, blk & 1u)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        tc_fence_after();
        const uint64_t k = uint64_t(stile) * kTcM + 32 * quad + lane;
        double* ps = a.part_sum + k * a.P_pad + uint64_t(ptile) * kTcN;
        uint32_t* pc = a.part_cnt + k * a.P_pad + uint64_t(ptile) * kTcN;
        const uint32_t lane_base = tmem + ((32 * quad) << 16);
#pragma unroll 1
        for (uint32_t cb = 0; cb < kTcN / 32; ++cb) {
          double acc[32];
#pragma unroll
          for (int i = 0; i < 32; ++i) acc[i] = 0.0;
          // limb planes of this pass's sum (the member plane, when present, is last)
          constexpr uint32_t kSum = COUNT_LAST ? uint32_t(NP) - 1u : uint32_t(NP);
#pragma unroll
          for (uint32_t j = 0; j < kSum; ++j) {
            uint32_t r[32];
            tmem_ld32(lane_base + j * kTcN + 32 * cb, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[i] += double(__uint_as_float(r[i]));
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) ps[32 * cb + i] += acc[i];
          if (COUNT_LAST) {
            uint32_t r[32];
            tmem_ld32(lane_base + (NP - 1) * kTcN + 32 * cb, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) pc[32 * cb + i] += __float2uint_rn(__uint_as_float(r[i]));
          }
        }
        tc_fence_before();
        mbar_arrive(accempty);
        ++blk;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---- 8-bit integer wide engine ---------------------------------------------------
// The wide GEMM of gnm_tc_accumulate with tcgen05.mma kind::i8: twice the MMA
// rate of BF16 per instruction, signed 8-bit weight limbs against unsigned
// 8-bit genotype operands (dosage 0/1/2 or the missing indicator), S32
// accumulators in tensor memory.  Every dosage weight of score k is split as
// l0 q0 + l1 q1 + l2 q2 + l3 q3 with q0 = max |x| of the score's values / 127,
// q(i+1) = q(i) / 254 and integers |l| <= 127 (each rounding leaves a
// remainder of at most half a quantum, which the next limb covers at 1/254 of
// that quantum), so the residual is below q3 / 2, 2^-31.9 of the score's
// largest value; missing corrections likewise.  (Three correction limbs,
// 2^-23.9, gave 5.4e-7 of the reference's 1e-6 tolerance on the biobank
// workload at full length.)  Products and
// their sums are exact integers in S32 for blocks of up to 2^23 variants; each
// plane's block sum reaches FP64 as int x its quantum at the flush, once per
// block (the flush's partial read-modify-write is one score row per lane, so
// flushing rarely keeps the memory queues free for the expansion).  Nine
// planes: dosage limbs 0-3, -correction limbs 0-3 and the member plane, in
// five passes (two planes fill tensor memory's 2 x 256 S32 columns; the
// member plane runs alone), each re-expanding the genotypes: dosage limbs
// 0-1 and 2-3 against the dosage operand, correction limbs 0-1 and 2-3 and
// the member plane against the missing indicator.  K = 128 variants per
// stage (a 128-byte K-major row), so a stage holds twice the variants of the
// BF16 kernel in the same bytes.
constexpr uint32_t kT8K = 128;       // variants per stage
// stages per flushed block: 2^23 variants, where |limb x dosage| <= 254 per
// variant keeps every S32 sum exact (254 x 2^23 < 2^31); an accumulate call
// shorter than that flushes once, at its end
constexpr uint32_t kT8Flush = (1u << 23) / kT8K;
constexpr int kT8Planes = 9;
constexpr uint32_t kT8Expand = 256;                 // expansion / epilogue threads (8 warps)
constexpr uint32_t kT8Threads = 64 + kT8Expand;     // + TMA warp + MMA warp
constexpr int kT8StagesPair = 4;   // TMA ring depth of two-plane passes (4 x 40 KB + 2 x 32 KB)
constexpr int kT8StagesOne = 6;    // of the one-plane pass (6 x 24 KB + 2 x 32 KB)

// ST: depth of the TMA ring (weight limbs + packed rows of a stage); the
// expanded genotype operand has its own two-deep ring, freed as soon as the
// stage's MMAs complete, so the TMA loads run ST stages ahead while the
// operand takes only two slots.
template <int NP, int ST>
struct T8Smem {
  static constexpr uint32_t kBStages = 2;
  static constexpr uint32_t kPlane = kTcM * kT8K;       // 16 KB
  static constexpr uint32_t kAStage = NP * kPlane;
  static constexpr uint32_t kB = kTcN * kT8K;           // 32 KB
  static constexpr uint32_t kPk = kT8K * (kTcN / 4);    // 8 KB
  static constexpr uint32_t kAOff = 0;
  static constexpr uint32_t kPkOff = kAOff + ST * kAStage;
  static constexpr uint32_t kBOff = kPkOff + ST * kPk;
  static constexpr uint32_t kBarOff = kBOff + kBStages * kB;
  static constexpr uint32_t kHolder = kBarOff + 8 * (2 * ST + 2 * kBStages + 2);
  static constexpr uint32_t kTotal = kHolder + 16 + 1024;  // + alignment slack
  static_assert(kTotal <= 227 * 1024, "shared memory");
  static_assert(kBOff % 1024 == 0 && kPkOff % 1024 == 0, "swizzled operands need 1 KB alignment");
};

struct T8Args {
  uint64_t num_rows;       // rows of this block
  int32_t a_x0;            // absolute variant index of block row 0 (multiple of 128)
  double* part_sum;
  uint32_t* part_cnt;
  uint64_t P_pad;
  uint64_t K_pad;
  const double* quanta;    // [kT8Planes][K_pad] quantum of every plane of every score
  uint32_t* err;
  uint32_t raster;         // 0: blockIdx.x = people tile, 1: blockIdx.x = score tile
  int32_t z0;              // first plane of this pass (TMA z coordinate)
};

// Sixteen 2-bit genotype codes -> sixteen 2-bit operand values in place: the
// allele-2 dosage (00 -> 0, 01 -> 0, 10 -> 1, 11 -> 2: low bit hi & ~lo, high
// bit hi & lo), or the missing indicator (01 -> 1).  Person q's values of
// four rows are then (w >> 2q) & 0x03030303, one per byte.
template <bool MISSING>
__device__ __forceinline__ uint32_t code_fields(uint32_t x) {
  const uint32_t hi = (x >> 1) & 0x55555555u, lo = x & 0x55555555u;
  return MISSING ? (lo & ~hi) : ((hi & ~lo) | ((hi & lo) << 1));
}

template <int NP, int ST, bool MISSING, bool COUNT_LAST>
__global__ void __launch_bounds__(kT8Threads, 1)
    gnm_t8_accumulate(const __grid_constant__ CUtensorMap amap,
                      const __grid_constant__ CUtensorMap pmap, T8Args a) {
  using L = T8Smem<NP, ST>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sb = smem_u32(smem);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ptile = a.raster ? blockIdx.y : blockIdx.x;
  const uint32_t stile = a.raster ? blockIdx.x : blockIdx.y;
  const uint32_t nit = uint32_t((a.num_rows + kT8K - 1) / kT8K);
  constexpr uint32_t BS = L::kBStages;
  auto full = [&](uint32_t s) { return sb + L::kBarOff + 8 * s; };          // TMA landed
  auto aempty = [&](uint32_t s) { return sb + L::kBarOff + 8 * (ST + s); }; // TMA slot free
  auto bready = [&](uint32_t b) { return sb + L::kBarOff + 8 * (2 * ST + b); };
  auto bempty = [&](uint32_t b) { return sb + L::kBarOff + 8 * (2 * ST + BS + b); };
  const uint32_t accfull = sb + L::kBarOff + 8 * (2 * ST + 2 * BS);
  const uint32_t accempty = sb + L::kBarOff + 8 * (2 * ST + 2 * BS + 1);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L::kHolder + 8);
  const uint32_t abort_addr = sb + L::kHolder + 8;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < ST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(aempty(s), 1);
    }
    for (uint32_t b = 0; b < BS; ++b) {
      mbar_init(bready(b), kT8Expand);
      mbar_init(bempty(b), 1);
    }
    mbar_init(accfull, 1);
    mbar_init(accempty, kT8Expand);
    *abort_flag = 0u;
    fence_mbar_init();
    prefetch_tmap(&amap);
    prefetch_tmap(&pmap);
  }
  if (warp == 1) {
    tmem_alloc(sb + L::kHolder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + L::kHolder);

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      for (uint32_t it = 0; it < nit; ++it) {
        const uint32_t s = it % ST, ph = (it / ST) & 1u;
        if (!mbar_wait_bounded(aempty(s), ph ^ 1u)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        if (lds_volatile_u32(abort_addr)) break;
        mbar_arrive_expect_tx(full(s), L::kAStage + L::kPk);
        tma_load_3d(sb + L::kAOff + s * L::kAStage, &amap, a.a_x0 + int32_t(it * kT8K),
                    int32_t(stile * kTcM), a.z0, full(s));
        tma_load_2d(sb + L::kPkOff + s * L::kPk, &pmap, int32_t(ptile * (kTcN / 4)),
                    int32_t(it * kT8K), full(s));
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_s8u8_s32(kTcM, kTcN);
      uint32_t blk = 0;
      for (uint32_t it = 0; it < nit; ++it) {
        const uint32_t s = it % ST;
        const uint32_t bsl = it % BS, bph = (it / BS) & 1u;
        const bool first = (it % kT8Flush) == 0;
        if (first && it > 0) {
          if (!mbar_wait_bounded(accempty, (blk - 1) & 1u)) {
            *abort_flag = 1u;
            atomicOr(a.err, kErrMmaTimeout);
            break;
          }
        }
        if (!mbar_wait_bounded(bready(bsl), bph)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        if (lds_volatile_u32(abort_addr)) break;
        tc_fence_after();
        const uint32_t a0 = sb + L::kAOff + s * L::kAStage;
        const uint32_t b0 = sb + L::kBOff + bsl * L::kB;
#pragma unroll
        for (uint32_t kk = 0; kk < kT8K / 32; ++kk) {   // K = 32 bytes per MMA
          const uint64_t bdesc = desc_kmajor_sw128(b0 + kk * 32);
#pragma unroll
          for (uint32_t j = 0; j < NP; ++j) {
            const uint64_t adesc = desc_kmajor_sw128(a0 + j * L::kPlane + kk * 32);
            tc_mma_i8(tmem + j * kTcN, adesc, bdesc, idesc, (first && kk == 0) ? 0u : 1u);
          }
        }
        tc_commit(aempty(s));
        tc_commit(bempty(bsl));
        if ((it % kT8Flush) == kT8Flush - 1 || it == nit - 1) {
          tc_commit(accfull);
          ++blk;
        }
      }
    }
  } else {
    // ---------------- genotype expansion + epilogue (warps 2-9) ----------------
    // warp 2 + 4h + vg: people half h (128 people), 16-variant chunks 2vg and
    // 2vg + 1; at block ends it drains TMEM lane quadrant warp % 4, column
    // blocks of its half
    const uint32_t ew = warp - 2;              // 0..7
    const uint32_t col = lane;                 // byte column: people 4col..4col+3
    const uint32_t vg = ew & 3;
    const uint32_t h = ew >> 2;
    const uint32_t quad = warp & 3;            // TMEM lane quadrant of this warp
    uint32_t blk = 0;
    for (uint32_t it = 0; it < nit; ++it) {
      const uint32_t s = it % ST, ph = (it / ST) & 1u;
      const uint32_t bsl = it % BS, bph = (it / BS) & 1u;
      if (!mbar_wait_bounded(full(s), ph)) {
        *abort_flag = 1u;
        atomicOr(a.err, kErrTmaTimeout);
        break;
      }
      // the operand slot is free once the MMAs of stage it - BS completed
      if (!mbar_wait_bounded(bempty(bsl), bph ^ 1u)) {
        *abort_flag = 1u;
        atomicOr(a.err, kErrMmaTimeout);
        break;
      }
      if (lds_volatile_u32(abort_addr)) break;
      const uint32_t pk = sb + L::kPkOff + s * L::kPk;
      const uint32_t bt = sb + L::kBOff + bsl * L::kB;
      {
        const uint32_t bc = 32 * h + col;   // byte column: people 4bc..4bc+3
#pragma unroll
        for (uint32_t cc = 0; cc < 2; ++cc) {
          const uint32_t c = 2 * vg + cc;   // 16-byte chunk (16 variants) of the operand row
          uint32_t x[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (uint32_t i = 0; i < 16; ++i)
            x[i >> 2] |= lds_u8(pk + (16 * c + i) * (kTcN / 4) + bc) << (8 * (i & 3));
#pragma unroll
          for (uint32_t i = 0; i < 4; ++i) x[i] = code_fields<MISSING>(x[i]);
#pragma unroll
          for (uint32_t q = 0; q < 4; ++q) {
            uint4 v;
            v.x = (x[0] >> (2 * q)) & 0x03030303u;
            v.y = (x[1] >> (2 * q)) & 0x03030303u;
            v.z = (x[2] >> (2 * q)) & 0x03030303u;
            v.w = (x[3] >> (2 * q)) & 0x03030303u;
            // operand row of person 128h + 4col + q (conflict-free 16-byte stores)
            const uint32_t n = 128 * h + 32 * q + col;
            sts_u128(bt + (n >> 3) * 1024 + (n & 7) * 128 + ((c ^ (n & 7)) << 4), v);
          }
        }
      }
      fence_proxy_async_smem();
      mbar_arrive(bready(bsl));

      if ((it % kT8Flush) == kT8Flush - 1 || it == nit - 1) {
        if (!mbar_wait_bounded(accfull, blk & 1u)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        tc_fence_after();
        const uint64_t k = uint64_t(stile) * kTcM + 32 * quad + lane;
        double* ps = a.part_sum + k * a.P_pad + uint64_t(ptile) * kTcN;
        uint32_t* pc = a.part_cnt + k * a.P_pad + uint64_t(ptile) * kTcN;
        const uint32_t lane_base = tmem + ((32 * quad) << 16);
        constexpr uint32_t kSum = COUNT_LAST ? uint32_t(NP) - 1u : uint32_t(NP);
        double qv[NP];
#pragma unroll
        for (uint32_t j = 0; j < uint32_t(NP); ++j) qv[j] = a.quanta[(a.z0 + j) * a.K_pad + k];
#pragma unroll 1
        for (uint32_t cb = h * (kTcN / 64); cb < (h + 1) * (kTcN / 64); ++cb) {
          if constexpr (kSum > 0) {
            double acc[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[i] = 0.0;
#pragma unroll
            for (uint32_t j = 0; j < kSum; ++j) {
              uint32_t r[32];
              tmem_ld32(lane_base + j * kTcN + 32 * cb, r);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 32; ++i) acc[i] = fma(double(int32_t(r[i])), qv[j], acc[i]);
            }
#pragma unroll
            for (int i = 0; i < 32; ++i) ps[32 * cb + i] += acc[i];
          }
          if (COUNT_LAST) {
            uint32_t r[32];
            tmem_ld32(lane_base + (NP - 1) * kTcN + 32 * cb, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) pc[32 * cb + i] += r[i];
          }
        }
        tc_fence_before();
        mbar_arrive(accempty);
        ++blk;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---- 8-bit wide engine on SM pairs ---------------------------------------------
// gnm_t8_accumulate with one tcgen05.mma.cta_group::2 spanning the two CTAs of
// a cluster: M = 256 scores (128 per CTA), N = 256 people (128 per CTA), K =
// 32 variants per instruction.  On one SM the N = 256 operand is read from
// shared memory once per plane and expanded by that SM alone, and the
// stage's shared-memory traffic (weight and genotype TMA writes, operand
// stores, MMA operand reads) takes longer than its MMAs; over a pair each SM
// stores, expands and serves only its 128 people, and each CTA's tensor
// memory still holds its 128 scores x all 256 people per plane.
//
// Roles per CTA: warp 0 issues the CTA's own TMA loads (its 128 scores' limb
// planes, its 128 people's packed rows) onto its own mbarriers; warps 2-9
// expand the CTA's genotypes into its half of the B operand and arrive (one
// lane per warp, after an async-proxy fence) on the even (leader) CTA's
// operand barrier, after the CTA's own TMA for the stage landed, so the
// arrival also vouches for its A half; warp 1 of the leader alone issues the
// MMAs, and its commits arrive on the freeing barriers of both CTAs
// (tcgen05.commit multicast).  Each CTA's epilogue drains its own 128 score
// rows; the leader waits for both epilogues before it overwrites the
// accumulators of the next block.  Every wait is bounded; a cluster barrier
// keeps both CTAs resident until neither can touch the other's shared
// memory, and tensor memory is allocated and released by warp 1 of both CTAs
// together.  The operand ring is four deep: every hand-off between the CTAs
// of a pair (operand ready, slot free) crosses SMs, so the expansion runs
// further ahead of the MMAs than on one SM.  The member plane's pass spans
// two score pairs per cluster (two planes' MMA work, like the other passes).
constexpr int kT8PairStagesPair = 4;  // TMA ring depth, two planes (4 x 36 KB + 4 x 16 KB)

template <int NP, int ST>
struct T8PairSmem {
  static constexpr uint32_t kBStages = 4;
  static constexpr uint32_t kPlane = kTcM * kT8K;         // 16 KB: 128 scores x 128 variants
  static constexpr uint32_t kAStage = NP * kPlane;
  static constexpr uint32_t kB = (kTcN / 2) * kT8K;       // 16 KB: this CTA's 128 people
  static constexpr uint32_t kPkRow = kTcN / 8;            // 32 packed bytes per variant row
  static constexpr uint32_t kPk = kT8K * kPkRow;          // 4 KB
  static constexpr uint32_t kAOff = 0;
  static constexpr uint32_t kPkOff = kAOff + ST * kAStage;
  static constexpr uint32_t kBOff = kPkOff + ST * kPk;
  static constexpr uint32_t kBarOff = kBOff + kBStages * kB;
  static constexpr uint32_t kHolder = kBarOff + 8 * (2 * ST + 2 * kBStages + 3);
  static constexpr uint32_t kTotal = kHolder + 16 + 1024;  // + alignment slack
  static_assert(kTotal <= 227 * 1024, "shared memory");
  static_assert(kBOff % 1024 == 0 && kPkOff % 1024 == 0, "swizzled operands need 1 KB alignment");
};

// One persistent launch per accumulate call: each cluster walks the work items
// w = cluster, cluster + clusters, ... of a static list, pass-major: passes
// 0-3 (dosage limbs 0-1 and 2-3, correction limbs 0-1 and 2-3) over every
// (people tile, score pair), then pass 4 (the member plane) over every
// (people tile, two score pairs).  Passes 1-3 add into FP64 partial arrays of
// their own, since a tile's passes may run on different clusters at the same
// time; pass 0 adds into the plan's partials with the other kernels, and the
// first call after a reset writes the pass arrays instead of adding to them.
struct T8PairArgs {
  uint64_t num_rows;       // rows of this block
  int32_t a_x0;            // absolute variant index of block row 0 (multiple of 128)
  double* part_sum;        // pass 0 (and every other kernel): [K_pad][P_pad]
  double* part_pass;       // passes 1-3: [3][K_pad][P_pad]
  uint32_t* part_cnt;
  uint64_t P_pad;
  uint64_t K_pad;
  const double* quanta;    // [kT8Planes][K_pad]
  uint32_t* err;
  uint32_t raster;         // 1: score pairs fastest within a pass
  uint32_t ptiles, spairs, spairs_m;   // people tiles, score pairs, pairs of score pairs
  uint32_t items;          // 4 * ptiles * spairs + ptiles * spairs_m
  uint32_t store;          // the pass arrays are written, not added to
};

struct PairItem {
  uint32_t pass, ptile, spair;   // pass 4: spair = index of the pair of score pairs
};

__device__ __forceinline__ PairItem pair_item(const T8PairArgs& a, uint32_t w) {
  const uint32_t per = a.ptiles * a.spairs;
  PairItem r;
  uint32_t t, sp;
  if (w < 4 * per) {
    r.pass = w / per;
    t = w % per;
    sp = a.spairs;
  } else {
    r.pass = 4;
    t = w - 4 * per;
    sp = a.spairs_m;
  }
  r.ptile = a.raster ? t / sp : t % a.ptiles;
  r.spair = a.raster ? t % sp : t / a.ptiles;
  return r;
}

template <int ST>
__global__ void __launch_bounds__(kT8Threads, 1)
    gnm_t8_pairs(const __grid_constant__ CUtensorMap amap2,
                 const __grid_constant__ CUtensorMap amap1,
                 const __grid_constant__ CUtensorMap pmap, T8PairArgs a) {
  using L = T8PairSmem<2, ST>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sb = smem_u32(smem);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();   // 0: leader (issues the MMAs), 1: peer
  const uint32_t cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;
  // this CTA's first score row of plane j of an item (uniform per CTA)
  auto srow = [&](const PairItem& w, uint32_t j) -> uint32_t {
    return w.pass == 4 ? (2 * (2 * w.spair + j) + rank) * kTcM : (2 * w.spair + rank) * kTcM;
  };
  const uint32_t nit = uint32_t((a.num_rows + kT8K - 1) / kT8K);
  constexpr uint32_t BS = L::kBStages;
  auto full = [&](uint32_t s) { return sb + L::kBarOff + 8 * s; };          // TMA landed
  auto aempty = [&](uint32_t s) { return sb + L::kBarOff + 8 * (ST + s); }; // TMA slot free
  auto bready = [&](uint32_t b) { return sb + L::kBarOff + 8 * (2 * ST + b); };
  auto bempty = [&](uint32_t b) { return sb + L::kBarOff + 8 * (2 * ST + BS + b); };
  const uint32_t accfull = sb + L::kBarOff + 8 * (2 * ST + 2 * BS);
  const uint32_t accempty = sb + L::kBarOff + 8 * (2 * ST + 2 * BS + 1);
  const uint32_t drain = sb + L::kBarOff + 8 * (2 * ST + 2 * BS + 2);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L::kHolder + 8);
  const uint32_t abort_addr = sb + L::kHolder + 8;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < ST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(aempty(s), 1);
    }
    for (uint32_t b = 0; b < BS; ++b) {
      mbar_init(bready(b), 2 * kT8Expand / 32);   // one arrival per expansion warp of both CTAs
      mbar_init(bempty(b), 1);
    }
    mbar_init(accfull, 1);
    mbar_init(accempty, 2 * kT8Expand);
    mbar_init(drain, 1);
    *abort_flag = 0u;
    fence_mbar_init();
    prefetch_tmap(&amap2);
    prefetch_tmap(&amap1);
    prefetch_tmap(&pmap);
  }
  if (warp == 1) {
    tmem_alloc_pair(sb + L::kHolder, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();   // barriers of both CTAs initialised, tensor memory allocated
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + L::kHolder);

  if (warp == 0) {
    // ---------------- TMA producer (each CTA its own halves) ----------------
    if (lane == 0) {
      uint32_t g = 0;   // stages issued so far, over every item
      bool stop = false;
      for (uint32_t wi = cid; wi < a.items && !stop; wi += ncl) {
        const PairItem w = pair_item(a, wi);
        for (uint32_t it = 0; it < nit; ++it, ++g) {
          const uint32_t s = g % ST, ph = (g / ST) & 1u;
          if (!mbar_wait_bounded(aempty(s), ph ^ 1u)) {
            *abort_flag = 1u;
            atomicOr(a.err, kErrMmaTimeout);
            stop = true;
            break;
          }
          if (lds_volatile_u32(abort_addr)) {
            stop = true;
            break;
          }
          mbar_arrive_expect_tx(full(s), L::kAStage + L::kPk);
          const uint32_t a_st = sb + L::kAOff + s * L::kAStage;
          const int32_t x = a.a_x0 + int32_t(it * kT8K);
          if (w.pass == 4) {   // the member plane of two score pairs
            tma_load_3d(a_st, &amap1, x, int32_t(srow(w, 0)), 8, full(s));
            tma_load_3d(a_st + L::kPlane, &amap1, x, int32_t(srow(w, 1)), 8, full(s));
          } else {
            tma_load_3d(a_st, &amap2, x, int32_t(srow(w, 0)), int32_t(2 * w.pass), full(s));
          }
          tma_load_2d(sb + L::kPkOff + s * L::kPk, &pmap,
                      int32_t(w.ptile * (kTcN / 4) + rank * L::kPkRow), int32_t(it * kT8K),
                      full(s));
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (leader CTA only) ----------------
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = idesc_s8u8_s32(2 * kTcM, kTcN);
      uint32_t g = 0, blk = 0;
      bool stop = false;
      for (uint32_t wi = cid; wi < a.items && !stop; wi += ncl) {
        for (uint32_t it = 0; it < nit; ++it, ++g) {
          const uint32_t s = g % ST;
          const uint32_t bsl = g % BS, bph = (g / BS) & 1u;
          const bool first = (it % kT8Flush) == 0;
          if (first && blk > 0) {
            // the epilogues of both CTAs drained the previous block
            if (!mbar_wait_bounded_cluster(accempty, (blk - 1) & 1u)) {
              *abort_flag = 1u;
              atomicOr(a.err, kErrMmaTimeout);
              stop = true;
              break;
            }
          }
          if (!mbar_wait_bounded(bready(bsl), bph)) {
            *abort_flag = 1u;
            atomicOr(a.err, kErrMmaTimeout);
            stop = true;
            break;
          }
          if (lds_volatile_u32(abort_addr)) {
            stop = true;
            break;
          }
          tc_fence_after();
          const uint32_t a0 = sb + L::kAOff + s * L::kAStage;
          const uint32_t b0 = sb + L::kBOff + bsl * L::kB;
#pragma unroll
          for (uint32_t kk = 0; kk < kT8K / 32; ++kk) {   // K = 32 bytes per MMA
            const uint64_t bdesc = desc_kmajor_sw128(b0 + kk * 32);
#pragma unroll
            for (uint32_t j = 0; j < 2; ++j) {
              const uint64_t adesc = desc_kmajor_sw128(a0 + j * L::kPlane + kk * 32);
              tc_mma_i8_pair(tmem + j * kTcN, adesc, bdesc, idesc,
                             (first && kk == 0) ? 0u : 1u);
            }
          }
          tc_commit_pair(aempty(s), 0x3);
          tc_commit_pair(bempty(bsl), 0x3);
          if ((it % kT8Flush) == kT8Flush - 1 || it == nit - 1) {
            tc_commit_pair(accfull, 0x3);
            ++blk;
          }
        }
      }
      // every MMA this thread issued has completed before either CTA moves on
      tc_commit_pair(drain, 0x1);
      if (!mbar_wait_bounded(drain, 0)) atomicOr(a.err, kErrMmaTimeout);
    }
  } else {
    // ---------------- genotype expansion + epilogue (warps 2-9) ----------------
    // warp 2 + e: 16-variant chunk e of the stage for the CTA's 128 people
    // (byte column `lane`: people 4 lane .. 4 lane + 3); at block ends it
    // drains TMEM lane quadrant warp % 4, column blocks of half e / 4
    const uint32_t ew = warp - 2;              // 0..7
    const uint32_t col = lane;
    const uint32_t c = ew;                     // 16-byte chunk (16 variants) of the operand row
    const uint32_t h = ew >> 2;
    const uint32_t quad = warp & 3;
    const uint32_t lead_accempty = mapa_shared(accempty, 0);
    const uint64_t pass_stride = a.K_pad * a.P_pad;
    uint32_t g = 0, blk = 0;
    bool stop = false;
    for (uint32_t wi = cid; wi < a.items && !stop; wi += ncl) {
      const PairItem w = pair_item(a, wi);
      const bool missing = w.pass >= 2;
      for (uint32_t it = 0; it < nit; ++it, ++g) {
        const uint32_t s = g % ST, ph = (g / ST) & 1u;
        const uint32_t bsl = g % BS, bph = (g / BS) & 1u;
        if (!mbar_wait_bounded(full(s), ph)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrTmaTimeout);
          stop = true;
          break;
        }
        // the operand slot is free once the MMAs of stage g - BS completed
        if (!mbar_wait_bounded(bempty(bsl), bph ^ 1u)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          stop = true;
          break;
        }
        if (lds_volatile_u32(abort_addr)) {
          stop = true;
          break;
        }
        const uint32_t pk = sb + L::kPkOff + s * L::kPk;
        const uint32_t bt = sb + L::kBOff + bsl * L::kB;
        {
          uint32_t x[4] = {0u, 0u, 0u, 0u};
#pragma unroll
          for (uint32_t i = 0; i < 16; ++i)
            x[i >> 2] |= lds_u8(pk + (16 * c + i) * L::kPkRow + col) << (8 * (i & 3));
#pragma unroll
          for (uint32_t i = 0; i < 4; ++i)
            x[i] = missing ? code_fields<true>(x[i]) : code_fields<false>(x[i]);
#pragma unroll
          for (uint32_t q = 0; q < 4; ++q) {
            uint4 v;
            v.x = (x[0] >> (2 * q)) & 0x03030303u;
            v.y = (x[1] >> (2 * q)) & 0x03030303u;
            v.z = (x[2] >> (2 * q)) & 0x03030303u;
            v.w = (x[3] >> (2 * q)) & 0x03030303u;
            // operand row of person 4col + q of this CTA's half; the pair's
            // TMEM column is 128 rank + row, the wide kernels' slot order
            const uint32_t n = 32 * q + col;
            sts_u128(bt + (n >> 3) * 1024 + (n & 7) * 128 + ((c ^ (n & 7)) << 4), v);
          }
        }
        // the warp's operand stores, fenced into the tensor core's (async)
        // proxy, are ordered before one arrival on the leader's barrier; its
        // consumer is the MMA, so no cluster-scope release is needed
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(mapa_shared(bready(bsl), 0));

        if ((it % kT8Flush) == kT8Flush - 1 || it == nit - 1) {
          if (!mbar_wait_bounded(accfull, blk & 1u)) {
            *abort_flag = 1u;
            atomicOr(a.err, kErrMmaTimeout);
            stop = true;
            break;
          }
          tc_fence_after();
          const uint32_t lane_base = tmem + ((32 * quad) << 16);
          if (w.pass == 4) {
#pragma unroll
            for (uint32_t j = 0; j < 2; ++j) {
              if (srow(w, j) >= a.K_pad) continue;
              const uint64_t k = uint64_t(srow(w, j)) + 32 * quad + lane;
              uint32_t* pc = a.part_cnt + k * a.P_pad + uint64_t(w.ptile) * kTcN;
#pragma unroll 1
              for (uint32_t cb = h * (kTcN / 64); cb < (h + 1) * (kTcN / 64); ++cb) {
                uint32_t r[32];
                tmem_ld32(lane_base + j * kTcN + 32 * cb, r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) pc[32 * cb + i] += r[i];
              }
            }
          } else if (srow(w, 0) < a.K_pad) {
            const uint64_t k = uint64_t(srow(w, 0)) + 32 * quad + lane;
            double* ps = (w.pass == 0 ? a.part_sum : a.part_pass + (w.pass - 1) * pass_stride) +
                         k * a.P_pad + uint64_t(w.ptile) * kTcN;
            // the pass arrays' first block after a reset is written, not added
            const bool write = w.pass > 0 && a.store && it < kT8Flush;
            const double q0 = a.quanta[(2 * w.pass) * a.K_pad + k];
            const double q1 = a.quanta[(2 * w.pass + 1) * a.K_pad + k];
#pragma unroll 1
            for (uint32_t cb = h * (kTcN / 64); cb < (h + 1) * (kTcN / 64); ++cb) {
              uint32_t r0[32], r1[32];
              tmem_ld32(lane_base + 32 * cb, r0);
              tmem_ld32(lane_base + kTcN + 32 * cb, r1);
              tmem_ld_wait();
              if (write) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  ps[32 * cb + i] = fma(double(int32_t(r1[i])), q1, double(int32_t(r0[i])) * q0);
              } else {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                  ps[32 * cb + i] += fma(double(int32_t(r1[i])), q1, double(int32_t(r0[i])) * q0);
              }
            }
          }
          tc_fence_before();
          mbar_arrive_cluster(lead_accempty);
          ++blk;
        }
      }
    }
  }
  tc_fence_before();
  __syncwarp();
  cluster_sync_all();   // no CTA leaves while the other may read or signal its shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem, 512);
  }
}

// 8-bit limb planes [kT8Planes][K_pad][V_pad] and their quanta [kT8Planes][K_pad]
// from the CSR: one thread per variant; the quanta by one thread per score.
__global__ void gnm_t8_quanta(const uint32_t* amax_bits, uint64_t K_pad, double* quanta) {
  const uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (k >= K_pad) return;
  const float am = __uint_as_float(amax_bits[k]);
  double q = am > 0.0f ? double(am) / 127.0 : 1.0;
  for (int l = 0; l < 4; ++l, q /= 254.0) {
    quanta[l * K_pad + k] = q;          // dosage limb l
    quanta[(4 + l) * K_pad + k] = q;    // correction limb l
  }
  quanta[8 * K_pad + k] = 1.0;          // member plane: counts
}

__global__ void gnm_t8_build_planes(const float* w, const float* corr, const uint32_t* cols,
                                    const uint64_t* offs, uint64_t V, const double* quanta,
                                    int8_t* planes, uint64_t K_pad, uint64_t V_pad) {
  const uint64_t v = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= V) return;
  const uint64_t plane = K_pad * V_pad;
  for (uint64_t e = offs[v]; e < offs[v + 1]; ++e) {
    const uint32_t k = cols[e];
    const uint64_t at = uint64_t(k) * V_pad + v;
    const double xs[2] = {double(w[e]), -double(corr[e])};
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      double r = xs[t];
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const double q = quanta[l * K_pad + k];
        const double li = fmin(fmax(rint(r / q), -127.0), 127.0);
        r -= li * q;
        planes[(4 * t + l) * plane + at] = int8_t(li);
      }
    }
    planes[8 * plane + at] = 1;
  }
}

// ---- narrow tensor engine (few score columns) ---------------------------------
// For a handful of scores the M = 128 score rows of gnm_tc_accumulate would be
// mostly empty, so the roles turn: M = 128 PEOPLE (TMEM lanes), N = 64 = the
// four limb planes of 16 scores (row n = 16 * plane + score, one 3D TMA box of
// the same limb planes), K = 64 variants per stage.  Each stage runs two MMAs
// per 16-variant slice: the dosage operand against the W' limbs and the
// missing-indicator operand against the -C limbs and the member plane, into
// 2 x 64 accumulator columns, so ONE pass produces sums and missing counts.
// The genotype expansion is the transposing one of gnm_tc_accumulate (operand
// row n = 32 q + col holds person 4 col + q), writing both operands, spread
// over eight warps (one 8-variant chunk per thread): with fewer, each warp's
// chain of dependent byte loads and permutes set the stage time.  Sums of a
// 16384-variant block are exact in FP32 (same limb argument) and are added to
// the FP64 partials of the CTA's variant split in natural person order at
// block ends; gnm_tc_finalize_slots adds the split slots in a fixed order.
constexpr uint32_t kNrM = 128;                // people per CTA
constexpr uint32_t kNrScores = 16;            // scores per CTA
constexpr uint32_t kNrN = 4 * kNrScores;      // accumulator columns per operand
constexpr uint32_t kNrStages = 4;
constexpr uint32_t kNrExpand = 256;           // expansion threads (warps 2-9)
constexpr uint32_t kNrThreads = 64 + kNrExpand;

struct NrSmem {
  static constexpr uint32_t kA = kNrM * kTcK * 2;          // 16 KB per operand
  static constexpr uint32_t kB = kNrN * kTcK * 2;          // 8 KB per limb set
  static constexpr uint32_t kPk = kTcK * (kNrM / 4);       // 2 KB packed rows
  static constexpr uint32_t kADos = 0;
  static constexpr uint32_t kAMis = kADos + kA;
  static constexpr uint32_t kBDos = kAMis + kA;
  static constexpr uint32_t kBMis = kBDos + kB;
  static constexpr uint32_t kPkOff = kBMis + kB;
  static constexpr uint32_t kStage = kPkOff + kPk;          // 50 KB
  static constexpr uint32_t kBarOff = kNrStages * kStage;
  static constexpr uint32_t kHolder = kBarOff + 8 * (3 * kNrStages + 2);
  static constexpr uint32_t kTotal = kHolder + 16 + 1024;   // + alignment slack
};
static_assert(NrSmem::kStage % 1024 == 0 && NrSmem::kBDos % 1024 == 0 &&
                  NrSmem::kBMis % 1024 == 0,
              "operand alignment");

struct NrArgs {
  uint64_t num_rows;          // rows of this block
  int32_t a_x0;               // absolute variant index of block row 0 (multiple of 64)
  uint32_t stages_per_split;  // 64-variant stages per blockIdx.z split
  double* part_sum;           // [split][K_pad][P_pad], natural person order
  uint32_t* part_cnt;
  uint64_t P_pad;
  uint64_t slot_stride;       // K_pad * P_pad
  uint32_t* err;
};

__global__ void __launch_bounds__(kNrThreads, 1)
    gnm_tc_narrow(const __grid_constant__ CUtensorMap dmap,
                  const __grid_constant__ CUtensorMap mmap,
                  const __grid_constant__ CUtensorMap pmap, NrArgs a) {
  using L = NrSmem;
  constexpr uint32_t ST = kNrStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sb = smem_u32(smem);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ptile = blockIdx.x, stile = blockIdx.y, split = blockIdx.z;
  const uint32_t nall = uint32_t((a.num_rows + kTcK - 1) / kTcK);
  const uint32_t it0 = split * a.stages_per_split;
  const uint32_t nit = it0 < nall ? min(a.stages_per_split, nall - it0) : 0u;
  auto full = [&](uint32_t s) { return sb + L::kBarOff + 8 * s; };
  auto bready = [&](uint32_t s) { return sb + L::kBarOff + 8 * (ST + s); };
  auto empty = [&](uint32_t s) { return sb + L::kBarOff + 8 * (2 * ST + s); };
  const uint32_t accfull = sb + L::kBarOff + 8 * (3 * ST);
  const uint32_t accempty = sb + L::kBarOff + 8 * (3 * ST + 1);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L::kHolder + 8);
  const uint32_t abort_addr = sb + L::kHolder + 8;
  if (nit == 0) return;   // a split past the block's last stage (uniform per CTA)

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < ST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(bready(s), kNrExpand);
      mbar_init(empty(s), 1);
    }
    mbar_init(accfull, 1);
    mbar_init(accempty, kNrExpand);
    *abort_flag = 0u;
    fence_mbar_init();
    prefetch_tmap(&dmap);
    prefetch_tmap(&mmap);
    prefetch_tmap(&pmap);
  }
  if (warp == 1) {
    tmem_alloc(sb + L::kHolder, 2 * kNrN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + L::kHolder);

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      for (uint32_t it = 0; it < nit; ++it) {
        const uint32_t s = it % ST, ph = (it / ST) & 1u;
        if (!mbar_wait_bounded(empty(s), ph ^ 1u)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        if (lds_volatile_u32(abort_addr)) break;
        const uint32_t st = sb + s * L::kStage;
        mbar_arrive_expect_tx(full(s), 2 * L::kB + L::kPk);
        const int32_t x = a.a_x0 + int32_t((it0 + it) * kTcK);
        tma_load_3d(st + L::kBDos, &dmap, x, int32_t(stile * kNrScores), 0, full(s));
        tma_load_3d(st + L::kBMis, &mmap, x, int32_t(stile * kNrScores), 0, full(s));
        tma_load_2d(st + L::kPkOff, &pmap, int32_t(ptile * (kNrM / 4)),
                    int32_t((it0 + it) * kTcK), full(s));
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_bf16_f32(kNrM, kNrN);
      uint32_t blk = 0;
      for (uint32_t it = 0; it < nit; ++it) {
        const uint32_t s = it % ST, ph = (it / ST) & 1u;
        const bool first = (it % kTcFlush) == 0;
        if (first && it > 0) {
          if (!mbar_wait_bounded(accempty, (blk - 1) & 1u)) {
            *abort_flag = 1u;
            atomicOr(a.err, kErrMmaTimeout);
            break;
          }
        }
        if (!mbar_wait_bounded(bready(s), ph)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        if (lds_volatile_u32(abort_addr)) break;
        tc_fence_after();
        const uint32_t st = sb + s * L::kStage;
#pragma unroll
        for (uint32_t kk = 0; kk < kTcK / 16; ++kk) {
          const uint32_t acc = (first && kk == 0) ? 0u : 1u;
          tc_mma_f16(tmem, desc_kmajor_sw128(st + L::kADos + kk * 32),
                     desc_kmajor_sw128(st + L::kBDos + kk * 32), idesc, acc);
          tc_mma_f16(tmem + kNrN, desc_kmajor_sw128(st + L::kAMis + kk * 32),
                     desc_kmajor_sw128(st + L::kBMis + kk * 32), idesc, acc);
        }
        tc_commit(empty(s));
        if ((it % kTcFlush) == kTcFlush - 1 || it == nit - 1) {
          tc_commit(accfull);
          ++blk;
        }
      }
    }
  } else {
    // ---------------- genotype expansion + epilogue (warps 2-9) ----------------
    const uint32_t pt = threadIdx.x - 64;   // 0..255
    const uint32_t col = pt & 31;           // byte column: people 4col..4col+3
    const uint32_t c = pt >> 5;             // 16-byte chunk: variants 8c..8c+7 of the stage
    const uint32_t quad = warp & 3;         // TMEM lane quadrant of this warp
    const uint32_t half = (warp - 2) >> 2;  // epilogue: scores 8 half .. 8 half + 7
    double* ps = a.part_sum + uint64_t(split) * a.slot_stride;
    uint32_t* pc = a.part_cnt + uint64_t(split) * a.slot_stride;
    uint32_t blk = 0;
    for (uint32_t it = 0; it < nit; ++it) {
      const uint32_t s = it % ST, ph = (it / ST) & 1u;
      if (!mbar_wait_bounded(full(s), ph)) {
        *abort_flag = 1u;
        atomicOr(a.err, kErrTmaTimeout);
        break;
      }
      if (lds_volatile_u32(abort_addr)) break;
      // explicit shared-space accesses: the realigned base is a generic pointer
      const uint32_t pk = sb + s * L::kStage + L::kPkOff;
      const uint32_t ad = sb + s * L::kStage + L::kADos;
      const uint32_t am = sb + s * L::kStage + L::kAMis;
      {
        const uint32_t r0 = 8 * c;
        uint32_t xl = 0, xh = 0;
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
          xl |= lds_u8(pk + (r0 + i) * (kNrM / 4) + col) << (8 * i);
          xh |= lds_u8(pk + (r0 + 4 + i) * (kNrM / 4) + col) << (8 * i);
        }
#pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
          const uint32_t yl = (xl >> (2 * q)) & 0x03030303u;
          const uint32_t yh = (xh >> (2 * q)) & 0x03030303u;
          uint4 vd, vm;
          vd.x = bf16_pair(yl & 0xFFFFu, kDosLo, kDosHi);
          vd.y = bf16_pair(yl >> 16, kDosLo, kDosHi);
          vd.z = bf16_pair(yh & 0xFFFFu, kDosLo, kDosHi);
          vd.w = bf16_pair(yh >> 16, kDosLo, kDosHi);
          vm.x = bf16_pair(yl & 0xFFFFu, kMisLo, kMisHi);
          vm.y = bf16_pair(yl >> 16, kMisLo, kMisHi);
          vm.z = bf16_pair(yh & 0xFFFFu, kMisLo, kMisHi);
          vm.w = bf16_pair(yh >> 16, kMisLo, kMisHi);
          // operand row of person 4col + q (conflict-free 16-byte stores)
          const uint32_t n = 32 * q + col;
          const uint32_t off = (n >> 3) * 1024 + (n & 7) * 128 + ((c ^ (n & 7)) << 4);
          sts_u128(ad + off, vd);
          sts_u128(am + off, vm);
        }
      }
      fence_proxy_async_smem();
      mbar_arrive(bready(s));

      if ((it % kTcFlush) == kTcFlush - 1 || it == nit - 1) {
        if (!mbar_wait_bounded(accfull, blk & 1u)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        tc_fence_after();
        // TMEM lane 32 quad + lane = operand row n -> person 4 (n % 32) + n / 32.
        // Column group g (16 columns): dosage limbs 0-3, -C limbs 0-2, member;
        // this thread reads its 8 scores of every group.
        const uint64_t person = uint64_t(ptile) * kNrM + 4 * lane + quad;
        const uint32_t lane_base = tmem + ((32 * quad) << 16) + 8 * half;
        double acc[8];
        uint32_t cnt[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) acc[k] = 0.0;
#pragma unroll
        for (uint32_t g = 0; g < 8; ++g) {
          uint32_t d[8];
          tmem_ld8(lane_base + 16 * g, d);
          tmem_ld_wait();
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k) {
            if (g < 7) acc[k] += double(__uint_as_float(d[k]));
            else cnt[k] = __float2uint_rn(__uint_as_float(d[k]));
          }
        }
        tc_fence_before();
        mbar_arrive(accempty);
        ++blk;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
          const uint64_t at = (uint64_t(stile) * kNrScores + 8 * half + k) * a.P_pad + person;
          ps[at] += acc[k];
          pc[at] += cnt[k];
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 2 * kNrN);
  }
}

// ---- people as M on 8-bit limbs ---------------------------------------------------
// Every score count on tcgen05.mma kind::i8 with people as M: the genotype
// operand A is expanded straight into TENSOR MEMORY, never into shared memory.
//
// What bounds it: with A in shared memory (the form this kernel replaced) a
// stage stored and re-read 64 KB of expanded operands per 128 people x 128
// variants, and shared-memory traffic, not the MMAs, set its time (tensor pipe
// 21 % busy).  Here the packed bytes are all that crosses shared memory:
//
//   * ldmatrix.m16n16.trans.b8 reads 16 variants x 16 packed bytes and hands
//     lane l the bytes of four consecutive variants, 4 (l % 4) ..., of byte
//     column l / 4 (and l / 4 + 8): one register is 4 variants x 4 people;
//   * per register, S = x >> 1 and D = x - ((x | S) & 0x55555555) give the
//     dosage fields (codes 00, 01, 10, 11 -> 0, 0, 1, 2); person q's operand word is
//     D & (0x03030303 << 2q) and its missing word x & ~S & (0x01010101 << 2q):
//     the field stays where it is, so person q's row is 4^q times its value,
//     and the epilogue's quantum takes 4^-q (a power of two: exact).  11
//     integer instructions per 16 genotypes and both operands;
//   * tcgen05.st.16x128b has the same fragment layout (lane l: TMEM row l / 4
//     and l / 4 + 8, 32-bit column l % 4), so the registers go to tensor memory
//     with no shuffle.  Byte column r of a warp's 8 is people 4r .. 4r + 3 on
//     TMEM lanes r, r + 8, r + 16, r + 24 of the warp's lane quadrant.
//
// Dosage limbs and correction limbs share their quanta (max over both), so
// both products add into the SAME 64 accumulator columns (limb j, score s:
// column 16 j + s), and the member plane gets 16 more: 80 columns per 128
// people.  That leaves room for NMT = 4 blocks of 128 people per CTA (320
// columns) beside a three-slot ring of operands (64 columns per 32 variants),
// and every 18 KB of limbs staged from L2 feeds 512 people instead of 128.
// NMT = 2 (256 people, eight slots) takes the cohorts and calls too small to
// fill the chip with 512-person tiles.  With 32 scores per CTA (NS = 2, the same
// 320 columns as 2 x 160, six slots) a genotype is expanded once for twice the
// scores: two tiles of 16 ran the expansion, which the MMAs of 16 scores do not
// cover, twice.
//
// Work is split evenly, not by tiles: first whole people tiles, all CTAs at the
// same stage, then of the last one to two tiles per CTA `quota` consecutive
// (people tile, stage) units each, so one CTA covers the tail of one tile and
// the head of the next and every SM finishes together; each of a tile's few
// segments writes its own FP64 slot.  CTAs of different score tiles walk the
// rows in step and share them in L2; whole tiles let the people tiles share the
// limbs too, which even shares alone, each at its own variants, read from HBM
// once they overflow L2 (200,000 people x 60,000 variants x 64 scores: 3.84 ms
// on 16 scores per CTA, 3.76 on 32, 3.39 on 32 with whole tiles, each a first pass;
// back to back the board's power limits it to 3.87).
//
// S32 sums are exact for 2^17 variants: |limb x 4^q x dosage| <= 127 x 128.
constexpr uint32_t kT8NrFlush = 1024;                // stages per exact S32 block (2^17 variants)
constexpr uint32_t kT8NrGroups = 4;                  // expansion warps per TMEM lane quadrant
constexpr uint32_t kT8NrThreads = 128 + 128 * kT8NrGroups;   // TMA, two MMA warps, one idle

template <int NMT, int NS>
struct T8NrSmem {
  static constexpr uint32_t kScores = kNrScores * NS;       // scores per CTA
  static constexpr uint32_t kRows = 4 * kScores;            // limb rows of the dosage operand
  static constexpr uint32_t kCols = 5 * kScores;            // accumulator columns per 128 people
  static constexpr uint32_t kStages = NS == 2 ? 5 : NMT == 4 ? 6 : 8;
  // operand ring, 32 variants each
  static constexpr uint32_t kSlots = NS == 2 ? 6 : NMT == 4 ? 3 : 8;
  static constexpr uint32_t kSlotCols = 16 * NMT;           // 8 dosage + 8 missing per block
  static constexpr uint32_t kParts = NMT / 2;               // a slot's parts: two blocks each
  static constexpr uint32_t kRing0 = kCols * NMT;           // first operand column
  static constexpr uint32_t kPeople = kNrM * NMT;
  static constexpr uint32_t kPkRow = kPeople / 4;           // packed bytes per variant row
  static constexpr uint32_t kPk = kT8K * kPkRow;
  static constexpr uint32_t kBDos = 0;                      // offsets inside a TMA stage
  static constexpr uint32_t kBMis = kRows * kT8K;           // 8 KB (NS = 1)
  static constexpr uint32_t kPkIn = kBMis + kCols * kT8K;   // + 10 KB
  static constexpr uint32_t kTma = kPkIn + kPk;             // 34, 26 or 44 KB
  static constexpr uint32_t kBarOff = kStages * kTma;
  static constexpr uint32_t kBars = 2 * kStages + 2 * kSlots * kParts + 4;
  static constexpr uint32_t kHolder = kBarOff + 8 * kBars;
  static constexpr uint32_t kTotal = kHolder + 16 + 1024;   // + alignment slack
  static_assert(kTotal <= 227 * 1024, "shared memory");
  static_assert(kTma % 1024 == 0 && kBMis % 1024 == 0 && kPkIn % 1024 == 0, "operand alignment");
  static_assert(kRing0 + kSlots * kSlotCols <= 512, "tensor memory columns");
};

// Slots of the narrow engine's partials that hold sums since the last reset, kept
// on the device so that a reset is one small memset and a captured call behaves
// as a plain one: a kernel writes the slots from `valid` on and adds to the
// others, and its last CTA (every CTA has read `valid` by then) moves `valid` up.
//   state[0] = valid, state[1] = CTAs of the running launch that are done
__device__ __forceinline__ void slots_written(uint32_t* state, uint32_t slots, uint32_t ctas) {
  __threadfence();
  if (atomicAdd(state + 1, 1u) == ctas - 1) {
    state[1] = 0u;
    if (state[0] < slots) state[0] = slots;
  }
}

// Zeroes slots valid .. slots - 1 ahead of a kernel that only adds.
__global__ void gnm_tc_open_slots(double* sum, uint32_t* cnt, uint64_t slot_stride,
                                  uint32_t slots, uint32_t* state) {
  const uint32_t valid = *reinterpret_cast<volatile uint32_t*>(state);
  const uint64_t end = uint64_t(slots) * slot_stride;
  for (uint64_t x = valid * slot_stride + uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; x < end;
       x += uint64_t(gridDim.x) * blockDim.x) {
    sum[x] = 0.0;
    cnt[x] = 0u;
  }
  __syncthreads();
  if (threadIdx.x == 0) slots_written(state, slots, gridDim.x);
}

struct T8NrArgs {
  int32_t a_x0;            // absolute variant index of block row 0 (multiple of 128)
  double* part_sum;        // [slots][K rounded to 16][P_pad]
  uint32_t* part_cnt;
  uint64_t P_pad;
  uint64_t slot_stride;    // elements per slot
  uint32_t* err;
  uint32_t stages;         // stages of the block (128 variants each)
  uint32_t ptiles;         // people tiles
  uint32_t rounds;         // whole people tiles per CTA, before its share of the rest
  uint32_t quota;          // (people tile, stage) units per share
  uint32_t slots;          // slots of every tile; those without a segment are zeroed
  uint32_t* state;         // {slots written since the reset, CTAs done}: see slots_written
  const double* quanta;    // [kT8Planes][K_pad]
  uint64_t K_pad;
  uint64_t K16;            // scores the partials hold
};

// The (people tile, stage) units of a CTA in order: `rounds` whole tiles, CTA c the
// tiles c, c + CTAs, ..., then units [u0, u1) of the tiles left.
struct T8NrWalk {
  uint32_t tile, st, round, units;   // the current unit; units in all
  uint32_t u0_tile, u0_st;
  __device__ explicit T8NrWalk(const T8NrArgs& a) {
    const uint32_t base = a.rounds * gridDim.x;
    const uint64_t rest = uint64_t(a.ptiles - base) * a.stages;
    const uint64_t u0 = min(uint64_t(blockIdx.x) * a.quota, rest);
    const uint64_t u1 = min(u0 + a.quota, rest);
    units = a.rounds * a.stages + uint32_t(u1 - u0);
    u0_tile = base + uint32_t(u0 / a.stages);
    u0_st = uint32_t(u0 % a.stages);
    round = 0;
    tile = a.rounds ? blockIdx.x : u0_tile;
    st = a.rounds ? 0u : u0_st;
  }
  __device__ void next(const T8NrArgs& a) {
    if (++st < a.stages) return;
    st = 0;
    if (round >= a.rounds) {
      ++tile;
    } else if (++round < a.rounds) {
      tile += gridDim.x;
    } else {
      tile = u0_tile;
      st = u0_st;
    }
  }
  // the slot of the current unit's segment: its share's place among the tile's
  __device__ uint32_t slot(const T8NrArgs& a) const {
    if (round < a.rounds) return 0u;
    const uint64_t t0 = uint64_t(tile - a.rounds * gridDim.x) * a.stages;
    return blockIdx.x - uint32_t(t0 / a.quota);
  }
};

template <int NMT, int NS>
__global__ void __launch_bounds__(kT8NrThreads, 1)
    gnm_t8_narrow(const __grid_constant__ CUtensorMap dmap,
                  const __grid_constant__ CUtensorMap mmap,
                  const __grid_constant__ CUtensorMap pmap, T8NrArgs a) {
  static_assert(NS == 1 || NMT == 2, "accumulator columns");
  using L = T8NrSmem<NMT, NS>;
  constexpr uint32_t ST = L::kStages, R = L::kSlots, RP = R * L::kParts;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sb = smem_u32(smem);
  const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t stile = blockIdx.y;
  T8NrWalk w(a);
  if (w.units == 0) {   // uniform per CTA
    if (threadIdx.x == 0) slots_written(a.state, a.slots, gridDim.x * gridDim.y);
    return;
  }
  auto full = [&](uint32_t s) { return sb + L::kBarOff + 8 * s; };           // TMA landed
  auto tempty = [&](uint32_t s) { return sb + L::kBarOff + 8 * (ST + s); };  // stage free
  // part p of operand slot b: filled by its four warps / read by its MMAs
  auto ready = [&](uint32_t b, uint32_t p) {
    return sb + L::kBarOff + 8 * (2 * ST + b * L::kParts + p);
  };
  auto sfree = [&](uint32_t b, uint32_t p) {
    return sb + L::kBarOff + 8 * (2 * ST + RP + b * L::kParts + p);
  };
  const uint32_t accfull = sb + L::kBarOff + 8 * (2 * ST + 2 * RP);
  const uint32_t accempty = accfull + 8, drain0 = accfull + 16;   // one drain per MMA warp
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L::kHolder + 8);
  const uint32_t abort_addr = sb + L::kHolder + 8;
  auto give_up = [&](uint32_t code) {
    *abort_flag = 1u;
    atomicOr(a.err, code);
  };

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < ST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(tempty(s), 2);   // both MMA warps
    }
    for (uint32_t b = 0; b < R; ++b)
      for (uint32_t p = 0; p < L::kParts; ++p) {
        mbar_init(ready(b, p), 4);
        mbar_init(sfree(b, p), 2 / L::kParts);
      }
    mbar_init(accfull, 2);
    mbar_init(accempty, 4 * kT8NrGroups);
    mbar_init(drain0, 1);
    mbar_init(drain0 + 8, 1);
    *abort_flag = 0u;
    fence_mbar_init();
    prefetch_tmap(&dmap);
    prefetch_tmap(&mmap);
    prefetch_tmap(&pmap);
  }
  if (warp == 1) {
    tmem_alloc(sb + L::kHolder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + L::kHolder);

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      uint32_t n = 0;            // stages issued
      bool ok = true;
      for (; n < w.units; ++n, w.next(a)) {
        const uint32_t s = n % ST, ph = (n / ST) & 1u;
        if (!mbar_wait_bounded(tempty(s), ph ^ 1u)) {
          give_up(kErrMmaTimeout);
          ok = false;
          break;
        }
        if (lds_volatile_u32(abort_addr)) {
          ok = false;
          break;
        }
        const uint32_t at = sb + s * L::kTma;
        mbar_arrive_expect_tx(full(s), L::kTma);
        const int32_t x = a.a_x0 + int32_t(w.st * kT8K);
        tma_load_2d(at + L::kPkIn, &pmap, int32_t(w.tile * L::kPkRow), int32_t(w.st * kT8K),
                    full(s));
        tma_load_3d(at + L::kBMis, &mmap, x, int32_t(stile * L::kScores), 4, full(s));
        tma_load_3d(at + L::kBDos, &dmap, x, int32_t(stile * L::kScores), 0, full(s));
      }
      if (!ok)   // nothing may still be in flight when the CTA exits (bounded)
        for (uint32_t i = n > ST ? n - ST : 0; i < n; ++i)
          mbar_wait_bounded(full(i % ST), (i / ST) & 1u);
    }
  } else if (warp == 1 || warp == 2) {
    // ---------------- MMA issuers ----------------
    // Warp 1 + i issues the MMAs of people blocks i NMT / 2 ...  Issue is what a
    // single warp runs out of: an MMA of these shapes takes 37 clocks, the
    // tensor core queues only a few, and each wait costs the warp about 90, so
    // one warp left the pipe idle for 40 % of a stage (2,000 clocks instead of
    // 1,200); two cover each other's waits.  Each whole warp runs the loop, with
    // votes for conditions, and one elected lane issues: addresses and
    // descriptors then stay in uniform registers, which tcgen05.mma reads (a
    // loop that only lane 0 runs moves each over per instruction: 60 clocks per
    // MMA).
    constexpr uint32_t idesc_d = idesc_u8s8_s32(kNrM, L::kRows);
    constexpr uint32_t idesc_m = idesc_u8s8_s32(kNrM, L::kCols);
    constexpr uint32_t kMine = NMT / 2;                  // blocks of this warp
    const uint32_t b0 = (warp - 1) * kMine;
    const uint32_t part = NMT == 4 ? warp - 1 : 0u;
    uint32_t blk = 0, inblk = 0, n = 0, slot = 0, sph = 0;
    const uint32_t utmem = __shfl_sync(0xFFFFFFFFu, tmem, 0);
    bool ok = true;
    for (; n < w.units && ok; ++n, w.next(a)) {
      const uint32_t s = n % ST;
      if (inblk == 0 && blk > 0 && !mbar_wait_warp(accempty, (blk - 1) & 1u)) {
        give_up(kErrMmaTimeout);
        ok = false;
        break;
      }
      const uint32_t at = sb + s * L::kTma;
      const uint64_t bm0 = desc_kmajor_sw128(at + L::kBMis);
      const uint64_t bd0 = desc_kmajor_sw128(at + L::kBDos);
      const bool last = w.st + 1 == a.stages || inblk + 1 == kT8NrFlush || n + 1 == w.units;
#pragma unroll
      for (uint32_t kk = 0; kk < kT8K / 32; ++kk) {   // 32 variants per slot and MMA
        // the warps that filled the slot waited for the stage's limbs too
        if (!mbar_wait_warp(ready(slot, part), sph)) {
          give_up(kErrMmaTimeout);
          ok = false;
          break;
        }
        tc_fence_after();
        if (elect_one()) {
          const uint64_t bm = bm0 + 2 * kk, bd = bd0 + 2 * kk;   // 32 bytes further
          const uint32_t op = utmem + L::kRing0 + slot * L::kSlotCols + 16 * b0;
          const uint32_t d = utmem + L::kCols * b0;
          // the missing product covers all columns, so it starts a block
          const uint32_t acc = (inblk == 0 && kk == 0) ? 0u : 1u;
#pragma unroll
          for (uint32_t t = 0; t < kMine; ++t)
            tc_mma_i8_ta(d + t * L::kCols, op + 16 * t + 8, bm, idesc_m, acc);
#pragma unroll
          for (uint32_t t = 0; t < kMine; ++t)
            tc_mma_i8_ta(d + t * L::kCols, op + 16 * t, bd, idesc_d, 1u);
          tc_commit(sfree(slot, part));
          if (kk == kT8K / 32 - 1) {
            tc_commit(tempty(s));
            if (last) tc_commit(accfull);
          }
        }
        __syncwarp();
        if (++slot == R) {
          slot = 0;
          sph ^= 1u;
        }
      }
      ++inblk;
      if (last) {   // end of a block
        ++blk;
        inblk = 0;
      }
    }
    // after a failure (this warp's or another's) the issued MMAs finish before the
    // CTA's memory goes (bounded)
    if (!ok) {
      const uint32_t drain = drain0 + 8 * (warp - 1);
      if (elect_one()) tc_commit(drain);
      __syncwarp();
      mbar_wait_bounded(drain, 0);
    }
  } else if (warp >= 4) {
    // ---------------- genotype expansion + epilogue (warps 4-19) ----------------
    const uint32_t quad = warp & 3;          // TMEM lane quadrant of this warp
    const uint32_t grp = (warp - 4) >> 2;    // 0..3
    // 512 people: a warp takes every second slot and half of its quadrant's
    // 32 packed bytes; 256 people: every fourth slot, all 16 bytes
    constexpr uint32_t kEvery = NMT == 4 ? 2 : 4;
    const uint32_t mine = NMT == 4 ? (grp & 1u) : grp;
    const uint32_t pairm = NMT == 4 ? (grp >> 1) : 0u;       // blocks 2 pairm, 2 pairm + 1
    const uint32_t chunk = (NMT / 2) * quad + pairm;         // 16-byte chunk of the row
    // this lane's ldmatrix row in the first of its slots (rows 32 apart keep
    // the swizzle's row bits), and the operand columns of the warp's blocks
    const uint32_t row = 32 * mine + lane;
    const uint32_t pk0 = sb + L::kPkIn + row * L::kPkRow +
                         ((NMT == 4 ? (chunk ^ (row & 7u)) : (chunk ^ ((row >> 1) & 3u))) << 4);
    const uint32_t op0 = tmem + ((32 * quad) << 16) + L::kRing0 + 32 * pairm;
    uint32_t blk = 0, inblk = 0, n = 0, slot = mine, sph = 0;
    bool first = true;   // the segment's first block
    const uint64_t valid = *reinterpret_cast<volatile uint32_t*>(a.state);
    for (; n < w.units; ++n, w.next(a)) {
      const uint32_t s = n % ST, ph = (n / ST) & 1u;
      // Waits that run out are remembered, not acted on: the tensor-memory stores
      // need the whole warp, and a vote per wait costs 10 % of the kernel.  The
      // stage's end leaves the loop for the warp as one.
      uint32_t late = mbar_wait_bounded(full(s), ph) ? 0u : kErrTmaTimeout;
      constexpr uint32_t kTurns = 4 / kEvery;   // this warp's slots of the stage
      uint32_t x[kTurns][4];   // [16 variants each][byte columns 0-7, 8-15]
#pragma unroll
      for (uint32_t j = 0; j < kTurns; ++j)
        ldmatrix_t_b8(pk0 + s * L::kTma + j * (32 * kEvery * L::kPkRow), x[j]);
      const uint32_t aborted = lds_volatile_u32(abort_addr);
#pragma unroll
      for (uint32_t j = 0; j < kTurns; ++j) {
        // columns of block h: dosage of variants 0-15, 16-31, missing likewise;
        // lo: people 0 and 1 of every byte, hi: people 2 and 3
        uint32_t lo[16], hi[16];
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
#pragma unroll
          for (uint32_t c = 0; c < 2; ++c) {
            const uint32_t xc = x[j][2 * c + h], sc = xc >> 1;
            const uint32_t dc = xc - ((xc | sc) & 0x55555555u);
            const uint32_t at = 8 * h + 2 * c;
            lo[at] = dc & 0x03030303u;
            lo[at + 1] = dc & 0x0C0C0C0Cu;
            hi[at] = dc & 0x30303030u;
            hi[at + 1] = dc & 0xC0C0C0C0u;
            lo[at + 4] = xc & ~sc & 0x01010101u;
            lo[at + 5] = xc & ~sc & 0x04040404u;
            hi[at + 4] = xc & ~sc & 0x10101010u;
            hi[at + 5] = xc & ~sc & 0x40404040u;
          }
        }
        // operands first, then the wait for their slot (the compiler would sink the
        // arithmetic below it)
#pragma unroll
        for (uint32_t i = 0; i < 16; ++i) asm volatile("" : "+r"(lo[i]), "+r"(hi[i]));
        if (!mbar_wait_bounded(sfree(slot, pairm), sph ^ 1u)) late |= kErrMmaTimeout;
        __syncwarp();
        tc_fence_after();
        const uint32_t op = op0 + slot * L::kSlotCols;
        tmem_st_16x128b_x8(op, lo);
        tmem_st_16x128b_x8(op + (16u << 16), hi);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ready(slot, pairm));
        slot += kEvery;
        if (slot >= R) {
          slot -= R;
          sph ^= 1u;
        }
      }
      if (__any_sync(0xFFFFFFFFu, (late | aborted) != 0u)) {
        if (late) give_up(late);
        break;
      }
      ++inblk;
      const bool tile_end = w.st + 1 == a.stages;
      if (tile_end || inblk == kT8NrFlush || n + 1 == w.units) {
        // ---- epilogue: drain one 128-person block of the tile ----
        inblk = 0;
        if (!mbar_wait_warp(accfull, blk & 1u)) {
          give_up(kErrMmaTimeout);
          break;
        }
        ++blk;
        tc_fence_after();
        const uint32_t t = grp % NMT;
        const uint32_t q = lane >> 3;        // row scale 4^q
        // TMEM lane 8q + r of quadrant `quad`, block t: person q of the
        // quadrant's packed byte 8t + r
        const uint64_t person = uint64_t(w.tile) * L::kPeople +
                                4 * (8 * NMT * quad + 8 * t + (lane & 7u)) + q;
        const uint32_t base = tmem + ((32 * quad) << 16) + t * L::kCols;
        const double scale = 1.0 / double(1u << (2 * q));
        const uint64_t sl = w.slot(a);
        const bool write = sl >= valid && first;
        const bool in = person < a.P_pad;
        // scores eight at a time; with 256 people two warps share a block's scores
        constexpr uint32_t kOcts = 2 * NS / (NMT == 4 ? 1 : 2);
#pragma unroll 1
        for (uint32_t i = 0; i < kOcts; ++i) {
          const uint32_t oct = NMT == 4 ? i : (grp >> 1) * kOcts + i;
          const uint64_t k0 = uint64_t(stile) * L::kScores + 8 * oct;
          if (k0 >= a.K16) break;   // (the same for the whole warp)
          double acc[8];
          uint32_t cnt[8];
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k) acc[k] = 0.0;
#pragma unroll
          for (uint32_t g = 0; g < 5; ++g) {
            uint32_t d[8];
            tmem_ld8(base + L::kScores * g + 8 * oct, d);
            tmem_ld_wait();
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) {
              if (g < 4)
                acc[k] = fma(double(int32_t(d[k])), a.quanta[g * a.K_pad + k0 + k] * scale, acc[k]);
              else
                cnt[k] = d[k] >> (2 * q);
            }
          }
          if (in) {
            double* ps = a.part_sum + sl * a.slot_stride + k0 * a.P_pad + person;
            uint32_t* pc = a.part_cnt + sl * a.slot_stride + k0 * a.P_pad + person;
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) {
              if (write) {
                ps[k * a.P_pad] = acc[k];
                pc[k * a.P_pad] = cnt[k];
              } else {
                ps[k * a.P_pad] += acc[k];
                pc[k * a.P_pad] += cnt[k];
              }
            }
            if (tile_end) {   // the tile's last segment: zero its unused new slots
              for (uint64_t z = sl + 1 > valid ? sl + 1 : valid; z < a.slots; ++z)
#pragma unroll
                for (uint32_t k = 0; k < 8; ++k) {
                  ps[(z - sl) * a.slot_stride + k * a.P_pad] = 0.0;
                  pc[(z - sl) * a.slot_stride + k * a.P_pad] = 0u;
                }
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(accempty);
        first = tile_end;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  if (threadIdx.x == 0) slots_written(a.state, a.slots, gridDim.x * gridDim.y);
}

// Limb planes from the CSR: one thread per variant.
// Per-score max(|w|, |corr|) as float bit patterns (non-negative floats order
// like their bits): shared-memory maxima per block, then one global atomic per
// score and block (global atomics only when the scores do not fit).
constexpr uint64_t kAmaxSharedScores = 8192;
__global__ void gnm_tc_amax(const float* w, const float* corr, const uint32_t* cols, uint64_t nnz,
                            uint64_t K_pad, uint32_t* amax_bits) {
  extern __shared__ uint32_t s_max[];
  const bool shared = K_pad <= kAmaxSharedScores;
  if (shared) {
    for (uint64_t k = threadIdx.x; k < K_pad; k += blockDim.x) s_max[k] = 0u;
    __syncthreads();
  }
  for (uint64_t e = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < nnz;
       e += uint64_t(gridDim.x) * blockDim.x) {
    const uint32_t m = __float_as_uint(fmaxf(fabsf(w[e]), fabsf(corr[e])));
    if (shared)
      atomicMax(s_max + cols[e], m);
    else
      atomicMax(amax_bits + cols[e], m);
  }
  if (shared) {
    __syncthreads();
    for (uint64_t k = threadIdx.x; k < K_pad; k += blockDim.x)
      if (s_max[k]) atomicMax(amax_bits + k, s_max[k]);
  }
}

__global__ void gnm_tc_build_planes(const float* w, const float* corr, const uint32_t* cols,
                                    const uint64_t* offs, uint64_t V, const uint32_t* amax_bits,
                                    __nv_bfloat16* dos, __nv_bfloat16* mis, uint64_t K_pad,
                                    uint64_t V_pad) {
  const uint64_t v = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= V) return;
  const uint64_t plane = K_pad * V_pad;
  for (uint64_t e = offs[v]; e < offs[v + 1]; ++e) {
    const uint32_t k = cols[e];
    // quantum q = 2^(E-8) with amax = f 2^E, f in [0.5, 1); then q/2^8, q/2^16,
    // q/2^24 (powers of two: the divisions are exact and every residual below
    // is exact in FP32)
    float q = 1.0f;
    const float am = __uint_as_float(amax_bits[k]);
    if (am > 0.0f) {
      int ex = 0;
      frexpf(am, &ex);
      q = ldexpf(1.0f, max(ex - 8, -125));   // q / 2^24 stays a (subnormal) FP32 value
    }
    const float qm = q * (1.0f / 256.0f), ql = q * (1.0f / 65536.0f),
                ql2 = q * (1.0f / 16777216.0f);
    const uint64_t at = uint64_t(k) * V_pad + v;
    const float xs[2] = {w[e], -corr[e]};
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const float x = xs[t];
      const float h = rintf(x / q) * q;
      const float r1 = x - h;
      const float m = rintf(r1 / qm) * qm;
      const float r2 = r1 - m;
      const float l = rintf(r2 / ql) * ql;
      __nv_bfloat16* base = t == 0 ? dos : mis;
      base[at] = __float2bfloat16_rn(h);
      base[plane + at] = __float2bfloat16_rn(m);
      base[2 * plane + at] = __float2bfloat16_rn(l);
      if (t == 0) base[3 * plane + at] = __float2bfloat16_rn(rintf((r2 - l) / ql2) * ql2);
    }
    mis[3 * plane + at] = __float2bfloat16_rn(1.0f);
  }
}

// out[o*K + k] = init[k] + the sum over the partials of person fam(o).  The
// partials are [score][person] and the output [person][score], so a CTA turns a
// block of 32 people in shared memory: its loads are consecutive people of one
// score, its stores consecutive scores of one person.  (One thread per output
// read a different cache line per thread: 2.02 ms against 0.46 ms on 100,000
// people x 512 scores, four FP64 arrays and the counts.)
//
// People as M: the slots written since the reset (`*state`) in person order, two at
// a time, four scores a thread (gnm_tc_finalize_slots, one score a thread, took 751
// us for two slots of 100,000 people x 512 scores, this 361).
// Wide kernels: one value in operand-row order, slot(f) = tile (f / 256), row
// 128*h + 32*(r%4) + (r%128)/4 with r = f % 256 and h = r / 128, plus the
// SM-pair kernel's partials of passes 1-3 (`pass`, may be null:
// [3][pass_stride]) in pass order.  Neither: the initial value.
constexpr uint32_t kFinTile = 32;

struct WideSums {          // the wide kernels' partials, sum null without any
  const double* sum;
  const uint32_t* cnt;
  const double* pass;      // passes 1-3 of the SM pairs, or null
  uint64_t P_pad, pass_stride;
  const uint32_t* opened;  // null, or zero while nothing was added (gnm_tc_open_wide)
};

// Zeroes the wide partials before the first block that adds to them since the
// reset, on a plan whose reset does not: state[2] says whether one did, so that
// captured blocks may replay in any order.
__global__ void gnm_tc_open_wide(double* sum, uint32_t* cnt, uint64_t n, uint32_t* state) {
  if (!*reinterpret_cast<volatile uint32_t*>(state + 2))
    for (uint64_t x = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; x < n;
         x += uint64_t(gridDim.x) * blockDim.x) {
      sum[x] = 0.0;
      cnt[x] = 0u;
    }
  __syncthreads();
  if (threadIdx.x == 0) {   // every CTA has read the flag once the last one counts
    __threadfence();
    if (atomicAdd(state + 1, 1u) + 1 == gridDim.x) {
      state[1] = 0u;
      state[2] = 1u;
    }
  }
}

struct SlotSums {          // people as M, sum null without any
  const double* sum;
  const uint32_t* cnt;
  uint64_t P_pad, stride;
  const uint32_t* state;   // slots written
};

__device__ __forceinline__ uint64_t wide_slot(uint64_t f) {
  const uint64_t r = f % kTcN, rr = r % 128;
  return f / kTcN * kTcN + 128 * (r / 128) + 32 * (rr % 4) + rr / 4;
}

__global__ void __launch_bounds__(256)
    gnm_tc_finalize(SlotSums slots, WideSums wide, const double* init,
                    const uint32_t* out_to_fam, uint64_t P, uint64_t K, uint32_t ktile0,
                    double* sums, uint32_t* counts) {
  __shared__ double s_sum[kFinTile][kFinTile + 1];
  __shared__ uint32_t s_cnt[kFinTile][kFinTile + 1];
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const uint64_t o0 = uint64_t(blockIdx.x) * kFinTile;
  const uint64_t k0 = uint64_t(ktile0 + blockIdx.y) * kFinTile;
  constexpr uint32_t kPer = kFinTile / 8;   // scores per warp
  const uint64_t o = o0 + lane;
  const uint64_t f = o >= P ? 0 : (out_to_fam ? out_to_fam[o] : o);
  double acc[kPer] = {};
  uint32_t cnt[kPer] = {};
  if (slots.sum && o < P) {
    const uint32_t n = *slots.state;
    const uint64_t first = (k0 + w) * slots.P_pad + f;
    for (uint32_t z = 0; z < n; z += 2) {
#pragma unroll
      for (uint32_t i = 0; i < kPer; ++i) {
        if (k0 + w + 8 * i >= K) break;
        const uint64_t at = z * slots.stride + first + 8 * i * slots.P_pad;
        acc[i] += slots.sum[at];
        cnt[i] += slots.cnt[at];
        if (z + 1 < n) {
          acc[i] += slots.sum[at + slots.stride];
          cnt[i] += slots.cnt[at + slots.stride];
        }
      }
    }
  }
  if (wide.sum && o < P && (!wide.opened || *wide.opened)) {
    const uint64_t first = (k0 + w) * wide.P_pad + wide_slot(f);
#pragma unroll
    for (uint32_t i = 0; i < kPer; ++i) {
      if (k0 + w + 8 * i >= K) break;
      const uint64_t at = first + 8 * i * wide.P_pad;
      acc[i] += wide.sum[at];
      cnt[i] += wide.cnt[at];
      if (wide.pass)
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j) acc[i] += wide.pass[j * wide.pass_stride + at];
    }
  }
#pragma unroll
  for (uint32_t i = 0; i < kPer; ++i) {
    s_sum[w + 8 * i][lane] = acc[i];
    s_cnt[w + 8 * i][lane] = cnt[i];
  }
  __syncthreads();
  const uint64_t k = k0 + lane;
  if (k >= K) return;
  const double base = init[k];
#pragma unroll
  for (uint32_t i = 0; i < kPer; ++i) {
    const uint32_t r = w + 8 * i;
    if (o0 + r < P) {
      sums[(o0 + r) * K + k] = base + s_sum[lane][r];
      counts[(o0 + r) * K + k] = s_cnt[lane][r];
    }
  }
}

// The same from many slots (a cohort of few people tiles).  A CTA takes 32 people x 8 scores; two warps share a score, even and odd slots
// four at a time, so the sum over a small cohort's many slots (48 of them: one
// per CTA that met the tile) is a few memory latencies, and its order is fixed.
// `wide` holds what blocks of the same run left in the wide partials.
constexpr uint32_t kSlotScores = 8, kSlotWarps = 2 * kSlotScores;
__global__ void __launch_bounds__(32 * kSlotWarps)
    gnm_tc_finalize_slots(SlotSums slots, WideSums wide, const double* init,
                          const uint32_t* out_to_fam, uint64_t P, uint64_t K, uint32_t ktile0,
                          double* sums, uint32_t* counts) {
  __shared__ double s_sum[kSlotWarps][33];
  __shared__ uint32_t s_cnt[kSlotWarps][33];
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
  const uint64_t o0 = uint64_t(blockIdx.x) * 32;
  const uint64_t k0 = uint64_t(ktile0 + blockIdx.y) * kSlotScores;
  const uint64_t o = o0 + lane, k = k0 + w % kSlotScores;
  const uint32_t nslots = *slots.state, part = w / kSlotScores;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  uint32_t cnt = 0;
  if (o < P && k < K) {
    const uint64_t f = out_to_fam ? out_to_fam[o] : o;
    const double* ps = slots.sum + k * slots.P_pad + f;
    const uint32_t* pc = slots.cnt + k * slots.P_pad + f;
    for (uint32_t z = part; z < nslots; z += 8) {
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i)
        if (z + 2 * i < nslots) {
          acc[i] += ps[(z + 2 * i) * slots.stride];
          cnt += pc[(z + 2 * i) * slots.stride];
        }
    }
    if (wide.sum && part == 0 && (!wide.opened || *wide.opened)) {
      const uint64_t at = k * wide.P_pad + wide_slot(f);
      acc[1] += wide.sum[at];
      cnt += wide.cnt[at];
      if (wide.pass)
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j) acc[1] += wide.pass[j * wide.pass_stride + at];
    }
  }
  s_sum[w][lane] = (acc[0] + acc[1]) + (acc[2] + acc[3]);
  s_cnt[w][lane] = cnt;
  __syncthreads();
  // thread -> (person, score), scores fastest
  if (threadIdx.x >= 32 * kSlotScores) return;
  const uint32_t ks = threadIdx.x % kSlotScores, p = threadIdx.x / kSlotScores;
  if (o0 + p >= P || k0 + ks >= K) return;
  const uint64_t x = (o0 + p) * K + k0 + ks;
  sums[x] = init[k0 + ks] + (s_sum[ks][p] + s_sum[ks + kSlotScores][p]);
  counts[x] = s_cnt[ks][p] + s_cnt[ks + kSlotScores][p];
}

// ---- backward: dW[v,k] = sum_p d(p,v) dS[p,k], dC[v,k] = -sum_{p missing} dS[p,k]
//
// A tcgen05 GEMM with the variants as M: D[v, n] = sum_p A[v, p] B[n, p].  A is
// the allele-2 dosage (missing -> 0) re-expanded from the packed rows into BF16
// by CUDA-core warps; a .bed row is already contiguous along people, so the
// K-major operand row of a variant is its own row, expanded in place (no
// transpose).  B holds dS split into four BF16 limbs per score (row
// n = 16 * limb + score): the hi/mid/lo/lo2 split of the forward planes, each
// limb an integer multiple of its quantum (q, q/2^8, q/2^16, q/2^24 with
// 2^E = 256 q >= max_p |dS[p,k]|) with |integer| <= 256, so products with
// d in {0,1,2} are exact and every partial sum stays exact in FP32 below
// 32768 people, where the accumulators are flushed to FP64.  The only error
// left is the limb residual (< 2^-33 of the score's largest |dS|).
//
// The missing-call term touches ~1% of the calls, so it is not a second GEMM:
// the thread that expands a variant row finds the row's code-01 calls with
// SWAR masks and adds that person's FP32 dS row (staged next to the limbs)
// into FP32 registers, flushed to FP64 every 4096 people (about 41 terms at
// 1% missing: the FP32 rounding stays below 3e-6 of the |dS| it sums, which
// is itself ~1% of the score's sum of |dS|).  Converting every term to FP64
// instead saturated the conversion pipe.
//
// CTA: 128 variants x 16 scores; people in stages of 64 (one 128-byte
// K-major operand row per variant).  Warp 0 issues TMA (packed rows
// [128 x 16 bytes], dS limbs [64 x 64] BF16 with 128-byte swizzle, FP32 dS
// [64 people x 16 scores]), warp 1 owns 64 TMEM columns and issues
// tcgen05.mma (M = 128, N = 64, K = 16), warps 2-9 expand genotypes: two
// threads per variant row (row 32 * (warp % 4) + lane, the TMEM lane the pair
// later drains; people 32 * half ..), each draining 8 of the 16 scores.  With
// one expanding warp per scheduler the chain of dependent permutes and stores
// set the stage time; with two, their latencies overlap.
constexpr uint32_t kBwM = 128;                    // variants per CTA (TMEM lanes)
constexpr uint32_t kBwScores = 16;                // scores per CTA
constexpr uint32_t kBwN = 4 * kBwScores;          // limb rows = accumulator columns
constexpr uint32_t kBwK = 64;                     // people per stage
constexpr uint32_t kBwStages = 6;
constexpr uint32_t kBwFlush = 512;                // stages per exact FP32 block (32768 people)
constexpr uint32_t kBwMissFlush = 64;             // stages per FP32 missing-term sum (4096 people)
constexpr uint32_t kBwExpand = 256;               // expansion threads (warps 2-9)
constexpr uint32_t kBwThreads = 64 + kBwExpand;

struct BwSmem {
  static constexpr uint32_t kA = kBwM * kBwK * 2;           // 16 KB dosage operand
  static constexpr uint32_t kB = kBwN * kBwK * 2;           // 8 KB dS limbs
  static constexpr uint32_t kPk = kBwM * (kBwK / 4);        // 2 KB packed rows
  static constexpr uint32_t kDs = kBwK * kBwScores * 4;     // 4 KB FP32 dS
  static constexpr uint32_t kAOff = 0;
  static constexpr uint32_t kBOff = kAOff + kA;
  static constexpr uint32_t kPkOff = kBOff + kB;
  static constexpr uint32_t kDsOff = kPkOff + kPk;
  static constexpr uint32_t kStage = kDsOff + kDs;           // 30 KB
  static constexpr uint32_t kBarOff = kBwStages * kStage;
  static constexpr uint32_t kHolder = kBarOff + 8 * (3 * kBwStages + 2);
  static constexpr uint32_t kTotal = kHolder + 16 + 1024;    // + alignment slack
  // end of kernel: both halves' FP64 missing sums [2][128][16], over stage 0-1
  static constexpr uint32_t kSwap = 2 * kBwM * kBwScores * 8;
};
static_assert(BwSmem::kStage % 1024 == 0 && BwSmem::kBOff % 1024 == 0, "operand alignment");
static_assert(BwSmem::kSwap <= BwSmem::kBarOff, "swap area");

struct BwArgs {
  uint64_t V, K;
  uint32_t nstages;   // people stages: P_pad / kBwK
  float* gw;
  float* gc;          // may be null
  uint32_t* err;
};

// Two BF16 dosages from two codes held in bytes 0 and 1 of y (bytes 2-3 ignored).
__device__ __forceinline__ uint32_t dos_pair(uint32_t y) {
  return __byte_perm(kDosLo, kDosHi, y * 0x11u + 0x4040u);
}

__global__ void __launch_bounds__(kBwThreads, 1)
    gnm_tc_backward(const __grid_constant__ CUtensorMap rmap,
                    const __grid_constant__ CUtensorMap bmap,
                    const __grid_constant__ CUtensorMap dmap, BwArgs a) {
  using L = BwSmem;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sb = smem_u32(smem);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t vtile = blockIdx.x, stile = blockIdx.y;
  const uint32_t nit = a.nstages;
  constexpr uint32_t ST = kBwStages;
  auto full = [&](uint32_t s) { return sb + L::kBarOff + 8 * s; };
  auto aready = [&](uint32_t s) { return sb + L::kBarOff + 8 * (ST + s); };
  auto empty = [&](uint32_t s) { return sb + L::kBarOff + 8 * (2 * ST + s); };
  const uint32_t accfull = sb + L::kBarOff + 8 * (3 * ST);
  const uint32_t accempty = sb + L::kBarOff + 8 * (3 * ST + 1);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L::kHolder + 8);
  const uint32_t abort_addr = sb + L::kHolder + 8;

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < ST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(aready(s), kBwExpand);
      mbar_init(empty(s), 1);
    }
    mbar_init(accfull, 1);
    mbar_init(accempty, kBwExpand);
    *abort_flag = 0u;
    fence_mbar_init();
    prefetch_tmap(&rmap);
    prefetch_tmap(&bmap);
    prefetch_tmap(&dmap);
  }
  if (warp == 1) {
    tmem_alloc(sb + L::kHolder, kBwN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + L::kHolder);

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      for (uint32_t it = 0; it < nit; ++it) {
        const uint32_t s = it % ST, ph = (it / ST) & 1u;
        if (!mbar_wait_bounded(empty(s), ph ^ 1u)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        if (lds_volatile_u32(abort_addr)) break;
        const uint32_t st = sb + s * L::kStage;
        mbar_arrive_expect_tx(full(s), L::kB + L::kPk + L::kDs);
        tma_load_2d(st + L::kPkOff, &rmap, int32_t(it * (kBwK / 4)), int32_t(vtile * kBwM),
                    full(s));
        tma_load_2d(st + L::kBOff, &bmap, int32_t(it * kBwK), int32_t(stile * kBwN), full(s));
        tma_load_2d(st + L::kDsOff, &dmap, int32_t(stile * kBwScores), int32_t(it * kBwK),
                    full(s));
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_bf16_f32(kBwM, kBwN);
      uint32_t blk = 0;
      for (uint32_t it = 0; it < nit; ++it) {
        const uint32_t s = it % ST, ph = (it / ST) & 1u;
        const bool first = (it % kBwFlush) == 0;
        if (first && it > 0) {
          if (!mbar_wait_bounded(accempty, (blk - 1) & 1u)) {
            *abort_flag = 1u;
            atomicOr(a.err, kErrMmaTimeout);
            break;
          }
        }
        if (!mbar_wait_bounded(aready(s), ph)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          break;
        }
        if (lds_volatile_u32(abort_addr)) break;
        tc_fence_after();
        const uint32_t a0 = sb + s * L::kStage + L::kAOff;
        const uint32_t b0 = sb + s * L::kStage + L::kBOff;
#pragma unroll
        for (uint32_t kk = 0; kk < kBwK / 16; ++kk)
          tc_mma_f16(tmem, desc_kmajor_sw128(a0 + kk * 32), desc_kmajor_sw128(b0 + kk * 32), idesc,
                     (first && kk == 0) ? 0u : 1u);
        tc_commit(empty(s));
        if ((it % kBwFlush) == kBwFlush - 1 || it == nit - 1) {
          tc_commit(accfull);
          ++blk;
        }
      }
    }
  } else {
    // ---------------- genotype expansion + epilogue (warps 2-9) ----------------
    const uint32_t quad = warp & 3;
    const uint32_t half = (warp - 2) >> 2;  // people 32 half .. of each stage; scores 8 half ..
    const uint32_t r = 32 * quad + lane;    // variant row of this thread and its TMEM lane
    double gwd[8], gcd[kBwScores];
    float gcf[kBwScores];   // missing term of the last <= kBwMissFlush stages
#pragma unroll
    for (uint32_t k = 0; k < kBwScores; ++k) {
      gcd[k] = 0.0;
      gcf[k] = 0.0f;
    }
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) gwd[k] = 0.0;
    bool ok = true;
    uint32_t blk = 0;
    for (uint32_t it = 0; it < nit; ++it) {
      const uint32_t s = it % ST, ph = (it / ST) & 1u;
      if (!mbar_wait_bounded(full(s), ph)) {
        *abort_flag = 1u;
        atomicOr(a.err, kErrTmaTimeout);
        ok = false;
        break;
      }
      if (lds_volatile_u32(abort_addr)) {
        ok = false;
        break;
      }
      const uint32_t st = sb + s * L::kStage;
      // words 2 half, 2 half + 1 of the row: people 32 half + 16 w' ..
      // explicit shared-space accesses: the realigned base is a generic pointer
      const uint2 x2 = lds_u64(st + L::kPkOff + r * (kBwK / 4) + 8 * half);
      const uint32_t xw[2] = {x2.x, x2.y};
      const uint32_t arow = st + L::kAOff + (r >> 3) * 1024 + (r & 7) * 128;
#pragma unroll
      for (uint32_t w = 0; w < 2; ++w) {
        // byte j of s_q = code of person 4j + q of the word
        const uint32_t x = xw[w];
        const uint32_t s0 = x & 0x03030303u, s1 = (x >> 2) & 0x03030303u;
        const uint32_t s2 = (x >> 4) & 0x03030303u, s3 = (x >> 6) & 0x03030303u;
#pragma unroll
        for (uint32_t h = 0; h < 2; ++h) {
          // 16-byte chunk c = people 8c..8c+7 of the stage (bytes 2h, 2h+1 of x)
          const uint32_t sa = 0x40u + 0x22u * h, sbb = 0x51u + 0x22u * h;
          uint4 v;
          v.x = dos_pair(__byte_perm(s0, s1, sa));
          v.y = dos_pair(__byte_perm(s2, s3, sa));
          v.z = dos_pair(__byte_perm(s0, s1, sbb));
          v.w = dos_pair(__byte_perm(s2, s3, sbb));
          const uint32_t c = 4 * half + 2 * w + h;
          sts_u128(arow + ((c ^ (r & 7)) << 4), v);
        }
      }
      // missing calls (code 01): add the person's FP32 dS row; bit 2i of m
      // is person 32 half + i
      uint64_t m = (uint64_t(xw[1] & ~(xw[1] >> 1) & 0x55555555u) << 32) |
                   (xw[0] & ~(xw[0] >> 1) & 0x55555555u);
      while (m) {
        const uint32_t b = 63u - __clzll(m);   // highest set bit: one find-leading-one
        m ^= uint64_t(1) << b;
        const uint32_t drow = st + L::kDsOff + (32 * half + b / 2) * (kBwScores * 4);
#pragma unroll
        for (uint32_t q = 0; q < kBwScores / 4; ++q) {
          const uint4 f = lds_u128(drow + 16 * q);
          gcf[4 * q + 0] += __uint_as_float(f.x);
          gcf[4 * q + 1] += __uint_as_float(f.y);
          gcf[4 * q + 2] += __uint_as_float(f.z);
          gcf[4 * q + 3] += __uint_as_float(f.w);
        }
      }
      if ((it % kBwMissFlush) == kBwMissFlush - 1 || it == nit - 1) {
#pragma unroll
        for (uint32_t k = 0; k < kBwScores; ++k) {
          gcd[k] += double(gcf[k]);
          gcf[k] = 0.0f;
        }
      }
      fence_proxy_async_smem();
      mbar_arrive(aready(s));

      if ((it % kBwFlush) == kBwFlush - 1 || it == nit - 1) {
        if (!mbar_wait_bounded(accfull, blk & 1u)) {
          *abort_flag = 1u;
          atomicOr(a.err, kErrMmaTimeout);
          ok = false;
          break;
        }
        tc_fence_after();
        // columns 16 j + 8 half + k: limb j of score 8 half + k
        const uint32_t lane_base = tmem + ((32 * quad) << 16) + 8 * half;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
          uint32_t d[8];
          tmem_ld8(lane_base + 16 * j, d);
          tmem_ld_wait();
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k) gwd[k] += double(__uint_as_float(d[k]));
        }
        tc_fence_before();
        mbar_arrive(accempty);
        ++blk;
      }
    }
    // The two halves of a row hold the missing term of different people: add
    // them in a fixed order through shared memory (stage buffers are idle: the
    // last accumulator commit followed every MMA, and every TMA was consumed).
    named_barrier(1, kBwExpand);
    double* swap = reinterpret_cast<double*>(smem);
#pragma unroll
    for (uint32_t k = 0; k < kBwScores; ++k) swap[(half * kBwM + r) * kBwScores + k] = gcd[k];
    named_barrier(1, kBwExpand);
    const uint64_t v = uint64_t(vtile) * kBwM + r;
    if (ok && !lds_volatile_u32(abort_addr) && v < a.V) {
#pragma unroll
      for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t kl = 8 * half + k;
        const uint64_t kk = uint64_t(stile) * kBwScores + kl;
        if (kk < a.K) {
          a.gw[v * a.K + kk] = float(gwd[k]);
          if (a.gc)
            a.gc[v * a.K + kk] =
                float(-(swap[r * kBwScores + kl] + swap[(kBwM + r) * kBwScores + kl]));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, kBwN);
  }
}

// ---- backward on 8-bit limbs -------------------------------------------------------
// G = d^T dS and C = -m^T dS as one tcgen05.mma kind::i8 pass: A = the dosage and
// the missing indicator of 128 variants (TMEM lanes), expanded straight into
// TENSOR MEMORY, B = dS split into four signed 8-bit limbs per score (row
// n = 16 * limb + score; q0 = max_p |dS[p,k]| / 127, q(j+1) = q(j) / 254, every
// |limb| <= 127, residual below 2^-31.9 of the score's largest |dS|), S32
// accumulators converted to FP64 with the quanta.
//
// What bounds it: the form this replaced stored the expanded dosage in shared
// memory, where the MMA read it back, and added the FP32 dS row of every
// missing call on CUDA cores, one dependent chain per row; tensor pipe 11 %
// busy.  Here a thread owns one variant row (its TMEM lane):
//
//   * 16 packed bytes (64 people) per shared load, rows swizzled by the TMA so
//     that eight lanes' loads fall in different banks;
//   * a word's 16 dosages D = x - ((x | x >> 1) & 0x55555555) and missing bits
//     M = x & ~(x >> 1) & 0x55555555 become four operand words each by a LEFT
//     shift and a mask: people q, q + 4, q + 8, q + 12 in the top bits of the
//     four bytes, 64 times their value (the quantum takes 2^-6).  Left shifts
//     and the subtraction are multiply-adds by constants, so they run on the FMA
//     pipe beside the masks on the integer pipe;
//   * gnm_bw_build8 lays dS out in that order of people, so nothing is
//     transposed; tcgen05.st.32x32b writes 64 people of both operands.
//
// Both operands meet the same limbs (two MMAs of N = 64 per 32 people, at least
// 32 clocks each: 0.22 ms at 20,000 x 200,000 x 16, where the whole call takes 0.44
// in a short run and 0.49 in a long one; the operand ring's latency takes the
// rest).  The dense missing product costs less than the sparse FP32 sums did (0.44
// against 1.55 ms); it is right to the limbs' step, and a score whose values are
// spread wider than that allows takes sparse sums in FP64 (bw_beyond_limbs).  256
// variants per CTA share each limb tile (2 x 128 accumulator columns + 256 of
// operand ring).  CTAs take equal shares of (variant tile,
// 512-person stage) units; a tile inside one share is written by its CTA, the
// segments of a tile that spans shares go through FP64 slots that gnm_bw_join
// adds in order.  S32 sums are exact for 2^17 people (127 x 2 x 64 each).
constexpr uint32_t kBw8K = 512;                      // people per stage
constexpr uint32_t kBw8Tile = 2 * kBwM;              // variants per CTA tile
constexpr uint32_t kBw8Stages = 3;
constexpr uint32_t kBw8Flush = (1u << 17) / kBw8K;   // stages per exact S32 block
constexpr uint32_t kBw8Slots = 4;                    // operand slots per 128 variants, 64 people each
constexpr uint32_t kBw8SlotCols = 32;                // 16 dosage + 16 missing columns
constexpr uint32_t kBw8AccCols = 2 * kBwN;           // G and C columns per 128 variants
constexpr uint32_t kBw8Threads = 128 + 512;          // TMA, two MMA warps, one idle; 16 expansion

struct Bw8Smem {
  static constexpr uint32_t kBox = kBwN * 128;               // 8 KB: limbs of 128 people
  static constexpr uint32_t kB = kBw8K / 128 * kBox;         // 32 KB
  static constexpr uint32_t kPkRow = kBw8K / 4;              // 128 packed bytes per variant
  static constexpr uint32_t kPk = kBw8Tile * kPkRow;         // 32 KB packed rows
  static constexpr uint32_t kPkOff = kB;
  static constexpr uint32_t kStage = kB + kPk;
  static constexpr uint32_t kBarOff = kBw8Stages * kStage;
  static constexpr uint32_t kBars = 2 * kBw8Stages + 4 * kBw8Slots + 4;
  static constexpr uint32_t kHolder = kBarOff + 8 * kBars;
  static constexpr uint32_t kTotal = kHolder + 16 + 1024;     // + alignment slack
  static_assert(kTotal <= 227 * 1024, "shared memory");
  static_assert(kStage % 1024 == 0 && kPkOff % 1024 == 0, "operand alignment");
  static constexpr uint32_t kRing0 = 2 * kBw8AccCols;
  static_assert(kRing0 + 2 * kBw8Slots * kBw8SlotCols <= 512, "tensor memory columns");
  static_assert(kBw8K / 64 == 2 * kBw8Slots, "a stage is two turns of the operand ring");
};

struct Bw8Args {
  uint64_t V, K, K16;
  uint32_t stages;         // 512-person stages
  uint32_t vtiles;         // 256-variant tiles
  uint32_t quota;          // (variant tile, stage) units per CTA
  const double* quanta;    // [4][K16]
  const uint32_t* sparse;  // [K16] scores whose C bw_missing_terms writes
  double* part;            // [score tiles][CTAs][2][G, C][256][16]: a CTA's first / last segment
  float* gw;
  float* gc;               // may be null (CORR false)
  uint32_t* err;
  const uint8_t* rows;     // packed rows and FP32 dS [people][K], for those
  uint64_t pitch;
  const float* ds;
  uint64_t people;
};

// The missing term of the scores of a tile that the limbs cannot hold (`sparse`):
// C[v, k] = -(sum of the dS values of the people missing at v), in FP64.  Every warp
// of the CTA takes variants of its own once the CTA's share of the products is
// done; these entries of C are written here alone.
//
// Latency bounds it (20 warps per SM): a lane reads 64 people's codes two steps
// ahead, a scan places the missing ones in the warp's list, and when that holds 256
// or the row ends, lanes take (person, score) pairs, 16 consecutive scores of two
// people, 16 values each in flight.  20,000 people x 20,000 variants x 16 scores,
// every dS a NaN: 0.21 ms for the whole step (25.1 with one thread per variant and
// score walking all people, 0.09 with finite scores); x 200,000: 1.56 ms (0.44).
constexpr uint32_t kBwList = 256 + 2048;
__device__ __noinline__ void bw_missing_terms(const uint8_t* rows, uint64_t pitch, uint64_t people,
                                              uint64_t V, const float* ds, uint32_t K,
                                              const uint32_t* sparse, uint64_t k0, uint32_t warp,
                                              uint32_t warps, uint32_t* list, float* gc) {
  const uint32_t lane = threadIdx.x & 31u, half = lane >> 4;
  const uint64_t k = k0 + (lane & 15u);
  const bool on = k < K && sparse[k] != 0u;
  const uint64_t bytes = (people + 3) / 4, step = uint64_t(gridDim.x) * warps;
  const uint32_t chunks = uint32_t((people + 2047) / 2048);
  const float* col = ds + k;
  // (variant, 2,048-person chunk) to load next, two ahead of the one in work
  uint64_t lv = uint64_t(blockIdx.x) * warps + warp;
  uint32_t lc = 0;
  auto load = [&] {   // this lane's 64 people
    const uint8_t* row = rows + lv * pitch;
    const uint64_t b0 = 512 * uint64_t(lc) + 16 * lane;
    uint4 q = make_uint4(0u, 0u, 0u, 0u);
    // rows start 16-byte aligned, and all but the last one's padding may be read
    if (lv < V && (b0 + 16 <= bytes || (b0 < bytes && lv + 1 < V))) {
      q = *reinterpret_cast<const uint4*>(row + b0);
    } else if (lv < V && b0 < bytes) {
      uint32_t x[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (uint32_t b = 0; b < 16; ++b)
        if (b0 + b < bytes) x[b / 4] |= uint32_t(row[b0 + b]) << (8 * (b % 4));
      q = make_uint4(x[0], x[1], x[2], x[3]);
    }
    if (++lc == chunks) {
      lc = 0;
      lv += step;
    }
    return q;
  };
  uint4 q0 = load(), q1 = load();
  for (uint64_t v = uint64_t(blockIdx.x) * warps + warp; v < V; v += step) {
    double acc = 0.0;
    uint32_t held = 0;
    for (uint32_t c = 0; c < chunks; ++c) {
      uint32_t m[4] = {q0.x, q0.y, q0.z, q0.w};
      q0 = q1;
      q1 = load();
      const uint64_t p0 = 2048 * uint64_t(c) + 64 * lane;
      uint32_t mine = 0;
#pragma unroll
      for (uint32_t w = 0; w < 4; ++w) {
        m[w] &= ~(m[w] >> 1) & 0x55555555u;
        const uint64_t p = p0 + 16 * w;        // padding past the last person may be code 01
        if (p + 16 > people) m[w] &= p < people ? (1u << (2 * uint32_t(people - p))) - 1u : 0u;
        mine += __popc(m[w]);
      }
      uint32_t at = mine;
#pragma unroll
      for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, at, d);
        if (lane >= d) at += y;
      }
      const uint32_t total = __shfl_sync(0xFFFFFFFFu, at, 31);
      at += held - mine;
#pragma unroll
      for (uint32_t w = 0; w < 4; ++w)
        for (uint32_t x = m[w]; x; x &= x - 1)
          list[at++] = uint32_t(p0) + 16 * w + (__ffs(x) - 1) / 2;
      held += total;
      if (held < 256 && c + 1 < chunks) continue;
      __syncwarp();
      for (uint32_t i = half; i < held; i += 32) {
        uint32_t p[16];
        float f[16];
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j) p[j] = list[min(i + 2 * j, held - 1)];
#pragma unroll
        for (uint32_t j = 0; j < 16; ++j)
          f[j] = on && i + 2 * j < held ? col[uint64_t(p[j]) * K] : 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < 16; j += 4)
          acc += (double(f[j]) + double(f[j + 1])) + (double(f[j + 2]) + double(f[j + 3]));
      }
      __syncwarp();
      held = 0;
    }
    acc += __shfl_xor_sync(0xFFFFFFFFu, acc, 16);
    if (on && half == 0) gc[v * K + k] = float(-acc);
  }
}

static_assert(kBw8Threads / 32 * kBwList * 4 <= Bw8Smem::kBarOff, "lists in the stage buffers");

// Elements of one segment slot of Bw8Args::part.
constexpr uint64_t kBw8SlotElems = 2 * uint64_t(kBw8Tile) * kBwScores;

// {-1, 4, 16, 64}: the subtraction and the left shifts of the expansion as integer
// multiply-adds; in constant memory, unknown at compile time, so that the
// compiler issues IMAD on the FMA pipe (see gnm_plain.cu).
__constant__ uint32_t c_bw[4] = {0xFFFFFFFFu, 4u, 16u, 64u};

template <bool CORR>
__global__ void __launch_bounds__(kBw8Threads, 1)
    gnm_t8_backward(const __grid_constant__ CUtensorMap rmap,
                    const __grid_constant__ CUtensorMap bmap, Bw8Args a) {
  using L = Bw8Smem;
  constexpr uint32_t ST = kBw8Stages, R = kBw8Slots;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sb = smem_u32(smem);
  const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const uint32_t stile = blockIdx.y;
  const uint64_t units = uint64_t(a.vtiles) * a.stages;
  const uint64_t u0 = uint64_t(blockIdx.x) * a.quota;
  const uint64_t u1 = u0 + a.quota < units ? u0 + a.quota : units;
  if (u0 >= u1) return;   // uniform per CTA (the host launches none such)
  auto full = [&](uint32_t s) { return sb + L::kBarOff + 8 * s; };
  auto tempty = [&](uint32_t s) { return sb + L::kBarOff + 8 * (ST + s); };
  // operand slot b of 128-variant block t: filled by its four warps / read by its MMAs
  auto ready = [&](uint32_t t, uint32_t b) { return sb + L::kBarOff + 8 * (2 * ST + t * R + b); };
  auto sfree = [&](uint32_t t, uint32_t b) {
    return sb + L::kBarOff + 8 * (2 * ST + (2 + t) * R + b);
  };
  const uint32_t accfull = sb + L::kBarOff + 8 * (2 * ST + 4 * R);
  const uint32_t accempty = accfull + 8, drain0 = accfull + 16;   // one drain per MMA warp
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(smem + L::kHolder + 8);
  const uint32_t abort_addr = sb + L::kHolder + 8;
  volatile uint32_t* any_sparse = reinterpret_cast<volatile uint32_t*>(smem + L::kHolder + 12);
  auto give_up = [&](uint32_t code) {
    *abort_flag = 1u;
    atomicOr(a.err, code);
  };

  if (threadIdx.x == 0) {
    for (uint32_t s = 0; s < ST; ++s) {
      mbar_init(full(s), 1);
      mbar_init(tempty(s), 2);   // both MMA warps
    }
    for (uint32_t t = 0; t < 2; ++t)
      for (uint32_t b = 0; b < R; ++b) {
        mbar_init(ready(t, b), 4);
        mbar_init(sfree(t, b), 1);
      }
    mbar_init(accfull, 2);
    mbar_init(accempty, 16);
    mbar_init(drain0, 1);
    mbar_init(drain0 + 8, 1);
    *abort_flag = 0u;
    fence_mbar_init();
    prefetch_tmap(&rmap);
    prefetch_tmap(&bmap);
  }
  if (warp == 1) {
    tmem_alloc(sb + L::kHolder, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + L::kHolder);

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      uint32_t n = 0;
      uint32_t tile = uint32_t(u0 / a.stages), st = uint32_t(u0 % a.stages);
      bool ok = true;
      for (uint64_t u = u0; u < u1; ++u, ++n) {
        const uint32_t s = n % ST, ph = (n / ST) & 1u;
        if (!mbar_wait_bounded(tempty(s), ph ^ 1u)) {
          give_up(kErrMmaTimeout);
          ok = false;
          break;
        }
        if (lds_volatile_u32(abort_addr)) {
          ok = false;
          break;
        }
        const uint32_t at = sb + s * L::kStage;
        mbar_arrive_expect_tx(full(s), L::kStage);
        tma_load_2d(at + L::kPkOff, &rmap, int32_t(st * L::kPkRow), int32_t(tile * kBw8Tile),
                    full(s));
#pragma unroll
        for (uint32_t j = 0; j < kBw8K / 128; ++j)
          tma_load_2d(at + j * L::kBox, &bmap, int32_t(st * kBw8K + 128 * j),
                      int32_t(stile * kBwN), full(s));
        if (++st == a.stages) {
          st = 0;
          ++tile;
        }
      }
      if (!ok)   // nothing may still be in flight when the CTA exits (bounded)
        for (uint32_t i = n > ST ? n - ST : 0; i < n; ++i)
          mbar_wait_bounded(full(i % ST), (i / ST) & 1u);
    }
  } else if (warp == 1 || warp == 2) {
    // ---------------- MMA issuers (see gnm_t8_narrow): warp 1 + t, block t ----------------
    constexpr uint32_t idesc = idesc_u8s8_s32(kBwM, kBwN);
    const uint32_t t = warp - 1;
    uint32_t st = uint32_t(u0 % a.stages), blk = 0, inblk = 0, n = 0;
    const uint32_t left = uint32_t(u1 - u0);
    const uint32_t utmem = __shfl_sync(0xFFFFFFFFu, tmem, 0);
    const uint32_t d = utmem + kBw8AccCols * t;
    bool ok = true;
    for (; n < left && ok; ++n) {
      const uint32_t s = n % ST;
      if (inblk == 0 && blk > 0 && !mbar_wait_warp(accempty, (blk - 1) & 1u)) {
        give_up(kErrMmaTimeout);
        ok = false;
        break;
      }
      const bool last = st + 1 == a.stages || inblk + 1 == kBw8Flush || n + 1 == left;
#pragma unroll
      for (uint32_t i = 0; i < kBw8K / 64; ++i) {   // 64 people per slot
        if (!mbar_wait_warp(ready(t, i % R), (i / R) & 1u)) {
          give_up(kErrMmaTimeout);
          ok = false;
          break;
        }
        tc_fence_after();
        if (elect_one()) {
          const uint64_t b0 = desc_kmajor_sw128(sb + s * L::kStage + (i / 2) * L::kBox) + 4 * (i % 2);
          const uint32_t op = utmem + L::kRing0 + (t * R + i % R) * kBw8SlotCols;
          const uint32_t acc = (inblk == 0 && i == 0) ? 0u : 1u;
#pragma unroll
          for (uint32_t kk = 0; kk < 2; ++kk) {
            tc_mma_i8_ta(d, op + 8 * kk, b0 + 2 * kk, idesc, kk ? 1u : acc);
            if (CORR) tc_mma_i8_ta(d + kBwN, op + 16 + 8 * kk, b0 + 2 * kk, idesc, kk ? 1u : acc);
          }
          tc_commit(sfree(t, i % R));
          if (i == kBw8K / 64 - 1) {
            tc_commit(tempty(s));
            if (last) tc_commit(accfull);
          }
        }
        __syncwarp();
      }
      ++inblk;
      if (++st == a.stages) st = 0;
      if (last) {
        ++blk;
        inblk = 0;
      }
    }
    if (!ok) {   // issued MMAs finish before the CTA's memory goes (bounded)
      const uint32_t drain = drain0 + 8 * t;
      if (elect_one()) tc_commit(drain);
      __syncwarp();
      mbar_wait_bounded(drain, 0);
    }
  } else if (warp == 3) {   // for the end, read while the others work
    const uint64_t k = uint64_t(stile) * kBwScores + lane;
    const bool on = CORR && lane < kBwScores && k < a.K && a.sparse[k] != 0u;
    const uint32_t any = __any_sync(0xFFFFFFFFu, on);
    if (lane == 0) *any_sparse = any;
  } else if (warp >= 4) {
    // ---------------- genotype expansion + epilogue (warps 4-19) ----------------
    const uint32_t quad = warp & 3;
    const uint32_t grp = (warp - 4) >> 2;
    const uint32_t t = grp & 1u, mine = grp >> 1;   // block; this warp takes every second slot
    const uint32_t r = kBwM * t + 32 * quad + lane;  // variant row of the tile
    const uint32_t pk0 = sb + L::kPkOff + r * L::kPkRow;
    const uint32_t op0 =
        tmem + ((32 * quad) << 16) + L::kRing0 + (t * R + mine) * kBw8SlotCols;
    const uint32_t ready0 = ready(t, mine), sfree0 = sfree(t, mine);
    uint32_t tile = uint32_t(u0 / a.stages), st = uint32_t(u0 % a.stages);
    uint32_t blk = 0, inblk = 0, n = 0;
    double acc[kBwScores];   // epilogue: G (mine 0) or C (mine 1) of this row
#pragma unroll
    for (uint32_t k = 0; k < kBwScores; ++k) acc[k] = 0.0;
    for (uint64_t u = u0; u < u1; ++u, ++n) {
      const uint32_t s = n % ST, ph = (n / ST) & 1u;
      // waits that run out are acted on at the stage's end (see gnm_t8_narrow)
      uint32_t late = mbar_wait_bounded(full(s), ph) ? 0u : kErrTmaTimeout;
      const uint32_t aborted = lds_volatile_u32(abort_addr);
      uint4 x4 = lds_u128(pk0 + s * L::kStage + ((mine ^ (r & 7u)) << 4));
#pragma unroll
      for (uint32_t j = 0; j < kBw8K / 128; ++j) {
        const uint32_t xw[4] = {x4.x, x4.y, x4.z, x4.w};
        if (j + 1 < kBw8K / 128)   // the next slot's 64 people
          x4 = lds_u128(pk0 + s * L::kStage + (((2 * (j + 1) + mine) ^ (r & 7u)) << 4));
        uint32_t v[32];
#pragma unroll
        for (uint32_t w = 0; w < 4; ++w) {
          const uint32_t x = xw[w], sh = x >> 1;
          const uint32_t d = ((x | sh) & 0x55555555u) * c_bw[0] + x;   // x - (...)
          v[4 * w + 0] = (d * c_bw[3]) & 0xC0C0C0C0u;
          v[4 * w + 1] = (d * c_bw[2]) & 0xC0C0C0C0u;
          v[4 * w + 2] = (d * c_bw[1]) & 0xC0C0C0C0u;
          v[4 * w + 3] = d & 0xC0C0C0C0u;
          if (CORR) {
            const uint32_t m = x & ~sh & 0x55555555u;
            v[16 + 4 * w + 0] = (m * c_bw[3]) & 0x40404040u;
            v[16 + 4 * w + 1] = (m * c_bw[2]) & 0x40404040u;
            v[16 + 4 * w + 2] = (m * c_bw[1]) & 0x40404040u;
            v[16 + 4 * w + 3] = m & 0x40404040u;
          }
        }
        // operands first, then the wait for their slot: the wait covers the MMAs of
        // two slots before, and the compiler would sink the arithmetic below it
#pragma unroll
        for (uint32_t i = 0; i < (CORR ? 32u : 16u); ++i) asm volatile("" : "+r"(v[i]));
        // a stage is two turns of the ring, so slots and phases are constants
        const uint32_t op = op0 + (2 * (j % 2)) * kBw8SlotCols;
        if (!mbar_wait_bounded(sfree0 + 16 * (j % 2), (j / 2) ^ 1u)) late |= kErrMmaTimeout;
        __syncwarp();
        tc_fence_after();
        if (CORR)
          tmem_st_32x32b_x32(op, v);
        else
          tmem_st_32x32b_x16(op, v);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ready0 + 16 * (j % 2));
      }
      if (__any_sync(0xFFFFFFFFu, (late | aborted) != 0u)) {
        if (late) give_up(late);
        break;
      }
      ++inblk;
      const uint32_t tile_now = tile;
      const bool tile_end = ++st == a.stages;
      if (tile_end) {
        st = 0;
        ++tile;
      }
      if (tile_end || inblk == kBw8Flush || u + 1 == u1) {
        inblk = 0;
        if (!mbar_wait_warp(accfull, blk & 1u)) {
          give_up(kErrMmaTimeout);
          break;
        }
        ++blk;
        tc_fence_after();
        if (CORR || mine == 0) {
          const uint32_t base = tmem + ((32 * quad) << 16) + t * kBw8AccCols + mine * kBwN;
          // -64 for C: the product is of the missing indicator, C its negative
          const double scale = mine ? -1.0 / 64.0 : 1.0 / 64.0;
#pragma unroll
          for (uint32_t j = 0; j < 4; ++j)
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
              uint32_t d[8];
              tmem_ld8(base + 16 * j + 8 * h, d);
              tmem_ld_wait();
#pragma unroll
              for (uint32_t k = 0; k < 8; ++k)
                acc[8 * h + k] =
                    fma(double(int32_t(d[k])),
                        a.quanta[j * a.K16 + uint64_t(stile) * kBwScores + 8 * h + k] * scale,
                        acc[8 * h + k]);
            }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(accempty);
        if (tile_end || u + 1 == u1) {   // the segment is complete
          const uint64_t t0 = uint64_t(tile_now) * a.stages;
          const uint64_t v = uint64_t(tile_now) * kBw8Tile + r;
          const uint64_t k0 = uint64_t(stile) * kBwScores;
          if (CORR || mine == 0) {
            if (t0 >= u0 && tile_end) {   // the whole tile is this CTA's
              float* out = mine ? a.gc : a.gw;
              if (v < a.V)
#pragma unroll
                for (uint32_t k = 0; k < kBwScores; ++k)
                  if (k0 + k < a.K && !(CORR && mine && a.sparse[k0 + k]))
                    out[v * a.K + k0 + k] = float(acc[k]);
            } else {   // slot 0: the tile began in an earlier share, 1: it goes on in the next
              const uint64_t cta = uint64_t(stile) * gridDim.x + blockIdx.x;
              double* ps = a.part + (2 * cta + (t0 >= u0 ? 1 : 0)) * kBw8SlotElems +
                           (uint64_t(mine) * kBw8Tile + r) * kBwScores;
#pragma unroll
              for (uint32_t k = 0; k < kBwScores; ++k) ps[k] = acc[k];
            }
          }
#pragma unroll
          for (uint32_t k = 0; k < kBwScores; ++k) acc[k] = 0.0;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  // the stage buffers are idle: every load was consumed, every MMA committed
  if (CORR && *any_sparse && !lds_volatile_u32(abort_addr))
    bw_missing_terms(a.rows, a.pitch, a.people, a.V, a.ds, uint32_t(a.K), a.sparse,
                     uint64_t(stile) * kBwScores, warp, kBw8Threads / 32,
                     reinterpret_cast<uint32_t*>(smem) + kBwList * warp, a.gc);
}

// Adds the segments of every variant tile that spans CTA shares, in share order.
// blockIdx.x = boundary between shares b and b + 1: the tile cut by it is joined
// by the first boundary that cuts it.
__global__ void __launch_bounds__(256) gnm_bw_join(Bw8Args a, uint32_t ctas) {
  const uint64_t cut = uint64_t(blockIdx.x + 1) * a.quota;   // first unit of share b + 1
  const uint64_t tile = cut / a.stages, t0 = tile * a.stages, t1 = t0 + a.stages;
  if (cut == t0 || cut - t0 > a.quota) return;   // no tile is cut / an earlier boundary cut it
  const uint64_t first = blockIdx.x, last = (t1 - 1) / a.quota;
  const uint32_t stile = blockIdx.y;
  const uint32_t ops = a.gc ? 2 : 1;
  for (uint32_t x = blockIdx.z * blockDim.x + threadIdx.x; x < ops * kBw8Tile * kBwScores;
       x += gridDim.z * blockDim.x) {
    const uint32_t op = x / (kBw8Tile * kBwScores), e = x % (kBw8Tile * kBwScores);
    const uint64_t v = tile * kBw8Tile + e / kBwScores;
    const uint64_t k = uint64_t(stile) * kBwScores + e % kBwScores;
    if (v >= a.V || k >= a.K) continue;
    const bool sparse = op && a.sparse[k] != 0u;   // (read beside the slots)
    double s = 0.0;
    for (uint64_t c = first; c <= last; ++c) {
      // the first share holds the tile as its last segment, the others as their first
      const uint64_t slot = 2 * (uint64_t(stile) * ctas + c) + (c == first ? 1 : 0);
      s += a.part[slot * kBw8SlotElems + uint64_t(op) * kBw8Tile * kBwScores + e];
    }
    if (!sparse) (op ? a.gc : a.gw)[v * a.K + k] = float(s);
  }
}

// Per-score max |dS| as float bit patterns (non-negative floats order like their
// bits) and, where `spread` is given, the count of non-zero values and the sum of
// their biased exponents: integers, so the same whatever the order.  A CTA takes
// `per` rows of up to 256 scores; a thread's score is fixed, so it keeps its own and
// adds them once.
struct BwSpread {
  unsigned long long* exps;   // [K16]
  uint32_t* count;            // [K16]
};
__global__ void __launch_bounds__(256)
    gnm_bw_amax(const float* g, uint64_t rows, uint64_t K, uint32_t per, uint32_t* amax_bits,
                BwSpread spread) {
  __shared__ uint32_t s_max[256], s_count[256], s_exps[256];
  const uint32_t k0 = blockIdx.y * 256, K32 = uint32_t(K);
  const uint32_t cols = min(K32 - k0, 256u);
  const uint32_t height = cols == 1 ? 256u : 256u / cols;
  const uint32_t r = cols == 1 ? threadIdx.x : threadIdx.x / cols, c = threadIdx.x - r * cols;
  const uint64_t r0 = uint64_t(blockIdx.x) * per;
  const uint32_t n = uint32_t(r0 + per < rows ? per : rows - r0);
  const float* at = g + r0 * K + k0 + c;
  uint32_t m = 0, count = 0, exps = 0;
  for (uint32_t p = r; p < n && r < height; p += 8 * height) {
    uint32_t v[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i)
      v[i] = p + i * height < n ? __float_as_uint(fabsf(at[uint64_t(p + i * height) * K32])) : 0u;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
      m = max(m, v[i]);
      count += v[i] != 0u;
      exps += v[i] >> 23;
    }
  }
  auto add = [&](uint32_t k) {
    atomicMax(amax_bits + k, m);
    if (spread.exps) {
      atomicAdd(spread.exps + k, static_cast<unsigned long long>(exps));
      atomicAdd(spread.count + k, count);
    }
  };
  if (cols == 1) {   // every thread has the same score
    m = __reduce_max_sync(0xFFFFFFFFu, m);
    count = __reduce_add_sync(0xFFFFFFFFu, count);
    exps = __reduce_add_sync(0xFFFFFFFFu, exps);
    if (m && threadIdx.x % 32 == 0) add(k0);
    return;
  }
  s_max[threadIdx.x] = s_count[threadIdx.x] = s_exps[threadIdx.x] = 0u;
  __syncthreads();
  if (m) {
    atomicMax(s_max + c, m);
    atomicAdd(s_count + c, count);
    atomicAdd(s_exps + c, exps);
  }
  __syncthreads();
  m = s_max[threadIdx.x];
  count = s_count[threadIdx.x];
  exps = s_exps[threadIdx.x];
  if (threadIdx.x < cols && m) add(k0 + threadIdx.x);
}

// A score whose missing term needs more than its limbs: an infinity or NaN, or values
// that lie, in the geometric mean, over 2^8 below the largest one.  The limbs'
// step is 2^-31.9 of the largest, so values 2^-8 of it keep FP32's 24 bits.  Worst
// error over 2,000 variants, of the sum of the |dS| added (20,000 people, 0.1 %
// missing; limbs, an FP32 sum of the values, now): normal dS 3.6e-8, 4.4e-8, 3.6e-8;
// one of 2^7 4.7e-8, 6.4e-8, 4.7e-8; one of 2^8 8.0e-8, 5.9e-8, 4.0e-8; one of 2^21
// 3.7e-4, 5.8e-8, 4.0e-8; t with 2 degrees 3.9e-8, 6.2e-8, 3.9e-8; Cauchy 4.5e-6,
// 9.7e-8, 5.2e-8; half of the people 2^-20 of the others 5.1e-4, 7.3e-8, 4.9e-8.
__device__ __forceinline__ uint32_t bw_beyond_limbs(float am, unsigned long long exps,
                                                    uint32_t count) {
  const unsigned long long top = __float_as_uint(am) >> 23;
  return !isfinite(am) || top * count > exps + 8ull * count ? 1u : 0u;
}

// dS [rows][K] -> 8-bit limb rows (tile t = k / 16: rows 64t + 16j + k % 16,
// limb j) of P_pad people each, and their quanta [4][K16]; zeros past the last
// person and score.  sparse[k]: limbs cannot hold the score (bw_beyond_limbs), its
// missing term is summed from the dS values themselves.  Person p of each 16 is stored at 4 (p % 4) + p / 4 % 4, the
// order in which gnm_t8_backward expands a packed word.  A CTA takes 32 people x
// 16 scores: it reads whole dS rows and writes 32 consecutive bytes of a limb row.
__global__ void __launch_bounds__(512)
    gnm_bw_build8(const float* g, uint64_t rows, uint64_t K, uint64_t K16, uint64_t P_pad,
                  const uint32_t* amax_bits, BwSpread spread, int8_t* planes, double* quanta,
                  uint32_t* sparse) {
  __shared__ float s_val[32][kBwScores + 1];
  const uint64_t p0 = uint64_t(blockIdx.x) * 32, k0 = uint64_t(blockIdx.y) * kBwScores;
  const uint32_t at = threadIdx.x % 32, ks = threadIdx.x / 32;   // stored position, score
  const uint32_t p = (at & 16u) + 4 * (at % 4) + at / 4 % 4;     // its person (an involution)
  const uint64_t k = k0 + ks;
  // every load ahead of the barrier
  const float am = k < K ? __uint_as_float(amax_bits[k]) : 0.0f;
  const bool first = blockIdx.x == 0 && at == 0;   // writes the score's quanta and flag
  const unsigned long long exps = first ? spread.exps[k] : 0ull;
  const uint32_t count = first ? spread.count[k] : 0u;
  {
    const uint32_t q = threadIdx.x / kBwScores, c = threadIdx.x % kBwScores;
    s_val[q][c] = (p0 + q < rows && k0 + c < K) ? g[(p0 + q) * K + k0 + c] : 0.0f;
  }
  __syncthreads();
  double q = am == 0.0f ? 1.0 : double(am) / 127.0;   // a NaN stays one
  if (first) sparse[k] = bw_beyond_limbs(am, exps, count);
  const uint64_t row0 = uint64_t(blockIdx.y) * kBwN + ks;
  double rem = double(s_val[p][ks]);
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j, q /= 254.0) {
    const double li = fmin(fmax(rint(rem / q), -127.0), 127.0);
    rem -= li * q;
    planes[(row0 + kBwScores * j) * P_pad + p0 + at] = int8_t(li);
    if (first) quanta[j * K16 + k] = q;
  }
}

// dS in output order -> fam order (zero for people outside the keep set).
__global__ void gnm_scatter_grad(const float* gs, const uint32_t* out_to_fam, uint64_t P,
                                 uint64_t K, float* gsf) {
  const uint64_t x = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (x >= P * K) return;
  const uint64_t o = x / K, k = x % K;
  gsf[uint64_t(out_to_fam[o]) * K + k] = gs[x];
}

// dS [rows][K] -> limb rows (tile t = k / 16: rows 64t + 16j + k % 16, limb j)
// of P_pad people each, and the FP32 copy [P_pad][K16] for the missing term;
// zeros past the last person and the last score.
__global__ void gnm_bw_build(const float* g, uint64_t rows, uint64_t K, uint64_t K16,
                             uint64_t P_pad, const uint32_t* amax_bits, __nv_bfloat16* planes,
                             float* ds) {
  const uint64_t x = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (x >= K16 * P_pad) return;
  const uint64_t p = x % P_pad, k = x / P_pad;
  const bool in = p < rows && k < K;
  const float val = in ? g[p * K + k] : 0.0f;
  ds[p * K16 + k] = val;
  // quantum q = 2^(E-8), 2^E > max |dS| of the score (no smaller than 2^-126)
  float q = 1.0f;
  if (k < K) {
    const float am = __uint_as_float(amax_bits[k]);
    if (am > 0.0f) {
      int e = 0;
      frexpf(am, &e);
      q = ldexpf(1.0f, max(e - 8, -126));
    }
  }
  const uint64_t row0 = (k / kBwScores) * kBwN + (k % kBwScores);
  float rem = val;
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j) {
    const float qj = q * ldexpf(1.0f, -8 * int(j));   // power of two: exact division
    const float limb = qj > 0.0f ? rintf(rem / qj) * qj : 0.0f;
    rem -= limb;
    planes[(row0 + kBwScores * j) * P_pad + p] = __float2bfloat16_rn(limb);
  }
}

// ---- host ------------------------------------------------------------------------

template <int NP, int ST, bool MISSING, bool COUNT_LAST>
static cudaError_t launch_tc(const CUtensorMap& amap, const CUtensorMap& pmap, const TcArgs& a,
                             uint32_t ptiles, uint32_t stiles, cudaStream_t s) {
  using L = TcSmem<NP, ST>;
  const cudaError_t e = raise_smem_limit(
      reinterpret_cast<const void*>(gnm_tc_accumulate<NP, ST, MISSING, COUNT_LAST>),
      int(L::kTotal));
  if (e != cudaSuccess) return e;
  const dim3 grid = a.raster ? dim3(stiles, ptiles) : dim3(ptiles, stiles);
  gnm_tc_accumulate<NP, ST, MISSING, COUNT_LAST><<<grid, kTcThreads, L::kTotal, s>>>(amap, pmap,
                                                                                     a);
  return cudaGetLastError();
}

template <int NP, int ST, bool MISSING, bool COUNT_LAST>
static cudaError_t launch_t8(const CUtensorMap& amap, const CUtensorMap& pmap, const T8Args& a,
                             uint32_t ptiles, uint32_t stiles, cudaStream_t s) {
  using L = T8Smem<NP, ST>;
  const cudaError_t e = raise_smem_limit(
      reinterpret_cast<const void*>(gnm_t8_accumulate<NP, ST, MISSING, COUNT_LAST>),
      int(L::kTotal));
  if (e != cudaSuccess) return e;
  const dim3 grid = a.raster ? dim3(stiles, ptiles) : dim3(ptiles, stiles);
  gnm_t8_accumulate<NP, ST, MISSING, COUNT_LAST><<<grid, kT8Threads, L::kTotal, s>>>(amap, pmap,
                                                                                     a);
  return cudaGetLastError();
}

// Persistent clusters of two CTAs along x (CTA 2i + r is rank r of cluster
// i): as many as can be resident at once, at most one per work item.
static uint32_t pair_clusters(int dev, uint32_t items) {
  static std::mutex mu;
  static int cached[64] = {};
  int n = 0;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64) n = cached[dev];
  }
  if (n == 0) {
    using L = T8PairSmem<2, kT8PairStagesPair>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2);
    cfg.blockDim = dim3(kT8Threads);
    cfg.dynamicSmemBytes = L::kTotal;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, gnm_t8_pairs<kT8PairStagesPair>, &cfg) != cudaSuccess ||
        n <= 0) {
      (void)cudaGetLastError();
      int sms = 0;
      check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev),
                 "cudaDeviceGetAttribute");
      n = std::max(1, sms / 2);
    }
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 0 && dev < 64) cached[dev] = n;
  }
  return std::max<uint32_t>(1, std::min<uint32_t>(uint32_t(n), items));
}

static void launch_t8_pairs(const CUtensorMap& amap2, const CUtensorMap& amap1,
                            const CUtensorMap& pmap, const T8PairArgs& a, int dev,
                            cudaStream_t s) {
  using L = T8PairSmem<2, kT8PairStagesPair>;
  const void* fn = reinterpret_cast<const void*>(gnm_t8_pairs<kT8PairStagesPair>);
  check_cuda(raise_smem_limit(fn, int(L::kTotal)), "8-bit pair shared memory");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pair_clusters(dev, a.items));
  cfg.blockDim = dim3(kT8Threads);
  cfg.dynamicSmemBytes = L::kTotal;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  check_cuda(cudaLaunchKernelEx(&cfg, gnm_t8_pairs<kT8PairStagesPair>, amap2, amap1, pmap, a),
             "8-bit pair launch");
}

static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      fail(GNM_ERR_COMPUTE, "cuTensorMapEncodeTiled is not available from the driver");
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// 4 limb planes [4][K_pad][V_pad]; a box holds `np` consecutive planes.
static CUtensorMap make_plane_map(const __nv_bfloat16* planes, uint64_t V_pad, uint64_t K_pad,
                                  uint32_t box_scores, uint32_t np) {
  CUtensorMap map;
  cuuint64_t dims[3] = {V_pad, K_pad, 4};
  cuuint64_t strides[2] = {V_pad * 2, K_pad * V_pad * 2};
  cuuint32_t box[3] = {kTcK, box_scores, np};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = tensor_map_encoder()(
      &map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(planes), dims,
      strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fail(GNM_ERR_COMPUTE, "cuTensorMapEncodeTiled failed for limb planes");
  return map;
}

// 8-bit limb planes [kT8Planes][K_pad][V_pad]; a box holds `rows` scores of `np`
// consecutive planes.
static CUtensorMap make_plane_map8(const int8_t* planes, uint64_t V_pad, uint64_t K_pad,
                                   uint32_t rows, uint32_t np) {
  CUtensorMap map;
  cuuint64_t dims[3] = {V_pad, K_pad, uint64_t(kT8Planes)};
  cuuint64_t strides[2] = {V_pad, K_pad * V_pad};
  cuuint32_t box[3] = {kT8K, rows, np};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = tensor_map_encoder()(
      &map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t*>(planes), dims, strides, box,
      estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fail(GNM_ERR_COMPUTE, "cuTensorMapEncodeTiled failed for 8-bit planes");
  return map;
}

// Row-major 2D map [rows][cols] (cols innermost; the row stride is cols
// elements, a multiple of 16 bytes).
static CUtensorMap make_2d_map(CUtensorMapDataType type, uint32_t elem_bytes, const void* base,
                               uint64_t cols, uint64_t rows, uint32_t box_cols,
                               uint32_t box_rows, CUtensorMapSwizzle swizzle, const char* what) {
  if ((cols * elem_bytes) % 16 != 0 || reinterpret_cast<uintptr_t>(base) % 16 != 0)
    fail(GNM_ERR_COMPUTE, std::string(what) + ": rows are not 16-byte aligned");
  CUtensorMap map;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * elem_bytes};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = tensor_map_encoder()(&map, type, 2, const_cast<void*>(base), dims, strides, box,
                                    estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fail(GNM_ERR_COMPUTE, std::string("cuTensorMapEncodeTiled failed for ") + what);
  return map;
}

// Variant splits of the narrow engine: enough CTAs for about four waves, then
// the count whose last wave is fullest (at most 16 splits, one stage each).
static uint32_t narrow_splits(uint64_t base_ctas, uint64_t stages, int sms) {
  uint32_t best = 1;
  double best_score = -1.0;
  for (uint32_t s = 1; s <= 16 && s <= std::max<uint64_t>(1, stages); ++s) {
    const uint64_t ctas = base_ctas * s;
    const uint64_t waves = (ctas + sms - 1) / sms;
    const double tail = double(ctas) / double(waves * uint64_t(sms));
    const double score = tail * std::min(1.0, double(ctas) / (4.0 * sms));
    if (score > best_score + 1e-9) {
      best_score = score;
      best = s;
    }
  }
  return best;
}

// CTAs per score tile, tiles of 16 * ns scores sharing the SMs.
static uint32_t narrow_ctas(const TensorPlan* t, uint64_t K, uint32_t ns) {
  const uint64_t stiles = (K + kNrScores * ns - 1) / (kNrScores * ns);
  return std::max<uint32_t>(1, uint32_t(t->sms / stiles));
}

// The longest a CTA works, in units of 16 scores x all people tiles: its scores over
// the CTAs that share them, times the waves of CTAs (more than one past one score
// tile per SM).
static double narrow_cost(const TensorPlan* t, uint64_t K, uint32_t ns) {
  const uint64_t tiles = (K + kNrScores * ns - 1) / (kNrScores * ns);
  const uint64_t ctas = narrow_ctas(t, K, ns);
  const uint64_t waves = (tiles * ctas + t->sms - 1) / t->sms;   // over one only past `sms` tiles
  return double(ns * waves) / double(ctas);
}
// 16-score groups per CTA.  32 scores halve the CTAs that expand the same rows
// (20,000 people x 100,000 variants x 32: 337 us on 16, 324 on 32; 20,000 x 40,000
// x 256: 1123 and 1034), unless 16 pad enough fewer scores per CTA in use: 15 %,
// the expansion's share (40 scores, 48 against 64 padded: 71 and 77 us at 3,000 x
// 60,000; 100 scores, 112 against 128: 493 and 484 us at 20,000 x 40,000; 4,000
// scores, 250 tiles of 16 in two waves against 125 in one: 24.2 and 25.2 ms at
// 50,000 x 20,000, 3,000 scores 23.7 and 21.6).
static uint32_t narrow_scores(const TensorPlan* t, uint64_t K) {
  if (K <= kNrScores) return 1;
  return 1.15 * narrow_cost(t, K, 1) < narrow_cost(t, K, 2) ? 1 : 2;
}

// Over 64 scores: people as M against SM pairs, the better wide kernel.  100,000
// people x 40,000 variants x 512 scores 10.0 against 12.2 ms, x 150,000 37-38
// against 39.4 ms, 8,000 x 40,000 x 512 0.99 against 1.04; with a last score tile
// to fill, 20,000 x 40,000 x 256, 1.03 against 1.53, 3,000 x 20,000 x 100, 61 against
// 882 us.  At 100,000 x 500,000 x 512 the 2.3 GB of limbs stream through L2 once per
// round of people tiles and the board throttles: 136-145 against 128-130 ms.  So
// pairs keep plans of over 1 GB of limbs whose scores nearly fill their 256.
//
// Pairs also keep the plans whose score tiles leave SMs without work: a CTA belongs
// to one score tile, so 75 to 95 tiles of 32 scores occupy little more than half of
// 148 SMs.  What a kernel pays for, in scores of a full GPU: people as M 16 x SMs per
// unit of narrow_cost, pairs 256 each.  Where people as M pay 1.5 times as much or
// more, pairs are as fast or faster (people against pairs, 50,000 x 20,000 and 100,000
// x 39,000): 2,400 scores, 1.85, 21.2 and 18.7, 77.8 and 60.5 ms; 3,000 scores, 1.54,
// 21.6 and 23.0, 84.8 and 73.0 ms; below, 4,800 scores, 1.46, 36.0 and 36.1 ms; 1,600
// scores, 1.32, 10.6 and 13.2, 39.1 and 42.9 ms; 1,000 scores, 1.16, 5.4 and 7.4,
// 20.0 and 24.3 ms.
constexpr uint32_t kGridY = 65535;   // rows of a grid
static bool prefers_people(const gnm_plan* p, const TensorPlan* t) {
  const uint64_t K256 = (p->K + 255) / 256 * 256, limbs = kT8Planes * p->K * p->V;
  if (limbs > (uint64_t(1) << 30) && 20 * K256 <= 23 * p->K) return false;
  const uint32_t ns = narrow_scores(t, p->K);
  if ((p->K + kNrScores * ns - 1) / (kNrScores * ns) > kGridY) return false;
  const double paid = 16.0 * t->sms * narrow_cost(t, p->K, ns);
  return t->stiles < 2 || paid < 1.5 * double(K256);
}

// Over 64 scores, the slots of people as M beside the wide partials.
static void alloc_slots(gnm_plan* p) {
  TensorPlan* t = p->tensor;
  const uint64_t n = uint64_t(t->nalloc) * t->nslot;
  void* sum = pool_alloc(p->device, n * 8, "cudaMalloc(slots)");
  void* cnt = nullptr;
  try {
    cnt = pool_alloc(p->device, n * 4, "cudaMalloc(slots)");
  } catch (...) {
    pool_free(sum);
    throw;
  }
  t->d_slot_sum = static_cast<double*>(sum);
  t->d_slot_cnt = static_cast<uint32_t*>(cnt);
  p->device_bytes += n * 12;
}

void tensor_plan_create(gnm_plan* p, const gnm_prep_view* prep, PhaseTrace* trace) {
  auto mark = [&](const char* what) {
    if (trace) trace->mark(what);
  };
  auto* t = new TensorPlan();
  p->tensor = t;
  t->K_pad = (p->K + kTcM - 1) / kTcM * kTcM;
  t->V_pad = std::max<uint64_t>(kTcK, (p->V + kTcK - 1) / kTcK * kTcK);
  t->ptiles = uint32_t(std::max<uint64_t>(1, (p->fam + kTcN - 1) / kTcN));
  t->stiles = uint32_t(t->K_pad / kTcM);
  t->P_pad = uint64_t(t->ptiles) * kTcN;
  t->can_narrow = p->K <= kNarrowMaxScores;
  t->narrow = t->can_narrow;
  int sms = 0;
  check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device),
             "cudaDeviceGetAttribute");
  t->sms = uint32_t(std::max(1, sms));
  t->people = t->can_narrow || prefers_people(p, t);
  // 8-bit limbs unless a shape says otherwise: 1.4x the BF16 limbs' speed in the
  // wide kernels on the batched workload, errors below 2.3e-7 at full length on
  // every workload
  t->i8 = true;
  // SM pairs when the plan fills pairs of 128-score tiles (with one tile the
  // pair's second CTA would hold no scores)
  t->pair = t->stiles >= 2;
  // score tiles fastest: the CTAs (clusters) running at once share a people
  // tile's packed rows (batched workload: 126.8 against 144.6 ms per step on
  // pairs, 159.4 against 165.7 on one SM)
  p->raster = 1;
  if (t->V_pad > (uint64_t(1) << 31)) fail(GNM_ERR_INVALID, "too many variants for the tensor engine");

  const uint64_t plane = t->K_pad * t->V_pad;
  auto alloc = [&](void** ptr, uint64_t bytes, const char* what) {
    *ptr = pool_alloc(p->device, bytes, what);
    p->device_bytes += bytes;
  };
  alloc(reinterpret_cast<void**>(&t->d_planes_dos), 4 * plane * 2, "cudaMalloc(limb planes)");
  alloc(reinterpret_cast<void**>(&t->d_planes_mis), 4 * plane * 2, "cudaMalloc(limb planes)");
  const uint64_t k16 = (p->K + kNrScores - 1) / kNrScores * kNrScores;
  const uint64_t base = ((p->fam + kNrM - 1) / kNrM) * (k16 / kNrScores);
  t->P_nar = std::max<uint64_t>(1, (p->fam + 4 * kNrM - 1) / (4 * kNrM)) * (4 * kNrM);
  t->nslot = k16 * t->P_nar;
  t->d_state = p->d_err + 1;   // cleared with the error word by every reset
  // a tile of S stages meets at most S / quota + 2 CTAs' shares, and quota >=
  // ptiles * S / (CTAs per score tile); after whole tiles, quota >= S
  t->nscores = narrow_scores(t, p->K);
  const uint64_t people = t->nscores == 2 ? 2 * kNrM : 4 * kNrM;   // of the widest tile in use
  t->nalloc = narrow_ctas(t, p->K, t->nscores) /
                  uint32_t(std::max<uint64_t>(1, (p->fam + people - 1) / people)) + 2;
  t->nslots8 = t->nalloc;
  uint64_t part_elems = t->K_pad * t->P_pad;
  if (t->can_narrow) {   // one buffer for either layout: a run uses one of the two
    t->nsplits = narrow_splits(base, t->V_pad / kTcK, std::max(1, sms));
    t->nalloc = std::max(t->nalloc, t->nsplits);
    part_elems = std::max(part_elems, uint64_t(t->nalloc) * t->nslot);
  }
  alloc(reinterpret_cast<void**>(&t->d_part_sum), part_elems * 8, "cudaMalloc(partials)");
  alloc(reinterpret_cast<void**>(&t->d_part_cnt), part_elems * 4, "cudaMalloc(partials)");
  t->d_slot_sum = t->d_part_sum;
  t->d_slot_cnt = t->d_part_cnt;
  if (!t->people) {   // SM pairs' passes 1-3 (written before being read)
    if (t->pair)
      alloc(reinterpret_cast<void**>(&t->d_part_pass), 3 * t->K_pad * t->P_pad * 8,
            "cudaMalloc(pass partials)");
  } else if (!t->can_narrow) {   // blocks that start off a 128-variant boundary add to the wide sums
    alloc_slots(p);
  }
  check_cuda(cudaMemset(t->d_planes_dos, 0, 4 * plane * 2), "memset planes");
  check_cuda(cudaMemset(t->d_planes_mis, 0, 4 * plane * 2), "memset planes");
  t->V_pad8 = std::max<uint64_t>(kT8K, (p->V + kT8K - 1) / kT8K * kT8K);
  const uint64_t plane8 = t->K_pad * t->V_pad8;
  alloc(reinterpret_cast<void**>(&t->d_planes8), kT8Planes * plane8, "cudaMalloc(8-bit planes)");
  alloc(reinterpret_cast<void**>(&t->d_quanta8), kT8Planes * t->K_pad * 8, "cudaMalloc(quanta)");
  check_cuda(cudaMemset(t->d_planes8, 0, kT8Planes * plane8), "memset planes");
  mark("  tensor: planes alloc");

  const uint64_t nnz = p->V ? prep->sparse_row_offsets[p->V] : 0;
  float *dw = nullptr, *dc = nullptr;
  uint32_t* dq = nullptr;
  uint32_t* dcol = nullptr;
  uint64_t* doff = nullptr;
  dw = static_cast<decltype(dw)>(
      pool_alloc(p->device, std::max<uint64_t>(1, nnz) * 4, "plane build inputs"));
  dc = static_cast<decltype(dc)>(
      pool_alloc(p->device, std::max<uint64_t>(1, nnz) * 4, "plane build inputs"));
  dcol = static_cast<decltype(dcol)>(
      pool_alloc(p->device, std::max<uint64_t>(1, nnz) * 4, "plane build inputs"));
  doff = static_cast<decltype(doff)>(
      pool_alloc(p->device, (p->V + 1) * 8, "plane build inputs"));
  dq = static_cast<uint32_t*>(pool_alloc(p->device, t->K_pad * 4, "plane build inputs"));
  struct Tmp {
    void* a[5];
    ~Tmp() {
      for (void* x : a) pool_free(x);
    }
  } tmp{{dw, dc, dcol, doff, dq}};
  if (nnz) {
    copy_to_device(dw, prep->sparse_weights, nnz * 4, 0);
    copy_to_device(dc, prep->sparse_missing_corrections, nnz * 4, 0);
    copy_to_device(dcol, prep->sparse_score_columns, nnz * 4, 0);
  }
  copy_to_device(doff, prep->sparse_row_offsets, (p->V + 1) * 8, 0);
  mark("  tensor: csr upload");
  // per-score quantum from max |x| over the score's values (on the device)
  check_cuda(cudaMemset(dq, 0, t->K_pad * 4), "memset");
  if (nnz) {
    const uint32_t smem = t->K_pad <= kAmaxSharedScores ? uint32_t(t->K_pad * 4) : 0u;
    const uint64_t blocks = std::min<uint64_t>((nnz + 255) / 256, 4096);
    gnm_tc_amax<<<uint32_t(blocks), 256, smem>>>(dw, dc, dcol, nnz, t->K_pad, dq);
    check_cuda(cudaGetLastError(), "weight maximum launch");
  }
  if (p->V) {
    gnm_tc_build_planes<<<uint32_t((p->V + 255) / 256), 256>>>(
        dw, dc, dcol, doff, p->V, dq, t->d_planes_dos, t->d_planes_mis, t->K_pad, t->V_pad);
    check_cuda(cudaGetLastError(), "plane build launch");
  }
  gnm_t8_quanta<<<uint32_t((t->K_pad + 255) / 256), 256>>>(dq, t->K_pad, t->d_quanta8);
  check_cuda(cudaGetLastError(), "quanta launch");
  if (p->V) {
    gnm_t8_build_planes<<<uint32_t((p->V + 255) / 256), 256>>>(
        dw, dc, dcol, doff, p->V, t->d_quanta8, t->d_planes8, t->K_pad, t->V_pad8);
    check_cuda(cudaGetLastError(), "8-bit plane build launch");
  }
  check_cuda(cudaStreamSynchronize(0), "plane build");
  mark("  tensor: plane build");
  t->map8_2 = make_plane_map8(t->d_planes8, t->V_pad8, t->K_pad, kTcM, 2);
  t->map8_1 = make_plane_map8(t->d_planes8, t->V_pad8, t->K_pad, kTcM, 1);
  t->map_dos = make_plane_map(t->d_planes_dos, t->V_pad, t->K_pad, kTcM, kTcPlanes);
  t->map_mis = make_plane_map(t->d_planes_mis, t->V_pad, t->K_pad, kTcM, kTcPlanes);
  t->nmap_dos = make_plane_map(t->d_planes_dos, t->V_pad, t->K_pad, kNrScores, 4);
  t->nmap_mis = make_plane_map(t->d_planes_mis, t->V_pad, t->K_pad, kNrScores, 4);
  t->nmap8_dos = make_plane_map8(t->d_planes8, t->V_pad8, t->K_pad, kNrScores * t->nscores, 4);
  t->nmap8_mis = make_plane_map8(t->d_planes8, t->V_pad8, t->K_pad, kNrScores * t->nscores, 5);
}

void tensor_plan_destroy(gnm_plan* p) {
  TensorPlan* t = p->tensor;
  if (!t) return;
  pool_free(t->d_planes_dos);
  pool_free(t->d_planes_mis);
  pool_free(t->d_planes8);
  pool_free(t->d_quanta8);
  if (t->d_slot_sum != t->d_part_sum) {
    pool_free(t->d_slot_sum);
    pool_free(t->d_slot_cnt);
  }
  pool_free(t->d_part_sum);
  pool_free(t->d_part_cnt);
  pool_free(t->d_part_pass);
  delete t;
  p->tensor = nullptr;
}

// The shape a plan starts with: 8-bit limbs with people as M (score tiles fastest,
// and over 64 scores the bit of SM pairs where the plan fills them).
uint32_t tensor_default_shape(const gnm_plan* p) {
  return p->tensor->can_narrow ? 7u : (p->tensor->stiles >= 2 ? 13u : 5u);
}
// The kernel that runs 8-bit blocks in a shape is gnm_t8_narrow: with the narrow bit
// (over 64 scores only beside kShapeExact), and over 64 scores in the default shape
// of a plan that prefers_people.  Every other shape with 8-bit limbs is the wide
// kernel its bits name.
static bool runs_people(const gnm_plan* p, uint32_t shape) {
  if (!(shape & 4u)) return false;
  return (shape & 2u) || (!p->tensor->can_narrow && p->tensor->people &&
                          shape == tensor_default_shape(p));
}
static bool people_as_m(const gnm_plan* p) { return runs_people(p, tensor_shape(p)); }
uint32_t tensor_people_shape(const gnm_plan* p) {
  return p->tensor->people ? tensor_default_shape(p) : kShapeExact | 7u;
}
uint32_t tensor_exact(const gnm_plan* p, uint32_t shape) {
  if (!(shape & 4u)) return shape;   // BF16 limbs have one code per kernel
  return kShapeExact | (runs_people(p, shape) ? 6u | (shape & 1u) : shape);
}

bool tensor_can_narrow(const gnm_plan* p) { return p->tensor && p->tensor->can_narrow; }
uint32_t tensor_shape(const gnm_plan* p) {
  const TensorPlan* t = p->tensor;
  return p->raster | (t->narrow || t->pinned_people ? 2u : 0u) | (t->i8 ? 4u : 0u) |
         (t->pair ? 8u : 0u) | t->exact;
}
void tensor_set_shape(gnm_plan* p, uint32_t shape) {
  TensorPlan* t = p->tensor;
  if ((shape & 2u) && !t->can_narrow && !(shape & kShapeExact))
    fail(GNM_ERR_INVALID, "the narrow tensor kernel serves at most 64 scores");
  const bool people = runs_people(p, shape);
  // what only some shapes need is allocated on first use
  if ((shape & 8u) && !people && !t->d_part_pass) {   // the SM-pair kernel's passes 1-3
    const uint64_t bytes = 3 * t->K_pad * t->P_pad * 8;
    t->d_part_pass = static_cast<double*>(pool_alloc(p->device, bytes, "pass partials"));
    p->device_bytes += bytes;
    t->pass_valid = false;
  }
  if (people && !t->can_narrow && t->d_slot_sum == t->d_part_sum) alloc_slots(p);
  t->narrow = (shape & 2u) != 0 && t->can_narrow;
  t->pinned_people = (shape & 2u) != 0 && !t->can_narrow;
  t->i8 = (shape & 4u) != 0;
  t->pair = (shape & 8u) != 0;
  t->exact = shape & kShapeExact;
  p->raster = shape & 1u;
}

// The wide partials start from zero; the narrow engine's slots are written, not
// added to, by the first call after the reset (slots_written).
static void clear_wide(TensorPlan* t, cudaStream_t s) {
  const uint64_t n = t->K_pad * t->P_pad;
  check_cuda(cudaMemsetAsync(t->d_part_sum, 0, n * 8, s), "reset partials");
  check_cuda(cudaMemsetAsync(t->d_part_cnt, 0, n * 4, s), "reset partials");
  t->wide_clear = true;
}

void tensor_reset(gnm_plan* p, cudaStream_t s) {
  TensorPlan* t = p->tensor;
  t->wide_clear = false;
  t->slots_used = false;
  if (!t->narrow && !people_as_m(p)) clear_wide(t, s);
  t->pass_valid = false;   // the next SM-pair accumulate writes its pass arrays
}

template <int NMT, int NS>
static void launch_t8_narrow(const gnm_plan* p, const uint8_t* d_rows, uint64_t pitch,
                             uint64_t nv, T8NrArgs a, cudaStream_t s) {
  using L = T8NrSmem<NMT, NS>;
  const TensorPlan* t = p->tensor;
  const CUtensorMap pmap =
      make_row_map(d_rows, p->bpv, nv, pitch, L::kPkRow, kT8K,
                   NMT == 4 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B);
  check_cuda(raise_smem_limit(reinterpret_cast<const void*>(gnm_t8_narrow<NMT, NS>),
                              int(L::kTotal)),
             "narrow 8-bit shared memory");
  const uint32_t ncta = narrow_ctas(t, p->K, NS);
  a.ptiles = uint32_t(std::max<uint64_t>(1, (p->bpv + L::kPkRow - 1) / L::kPkRow));
  // Whole tiles while at least two rounds of CTAs are left: those CTAs start every
  // tile at its first variant together and share the limbs in L2, which long rows'
  // limbs overflow (50,000 x 100,000 x 512, 460 MB of them: 15.2 ms with shares
  // only).  The one to two rounds that remain go in even shares.
  a.rounds = a.ptiles >= 2 * ncta ? a.ptiles / ncta - 1 : 0u;
  const uint64_t units = uint64_t(a.ptiles - a.rounds * ncta) * a.stages;
  a.quota = uint32_t((units + ncta - 1) / ncta);
  a.slots = (a.stages + a.quota - 2) / a.quota + 1;
  if (a.slots > t->nalloc) fail(GNM_ERR_COMPUTE, "narrow engine: more slots than allocated");
  const dim3 grid(a.rounds ? ncta : uint32_t((units + a.quota - 1) / a.quota),
                  uint32_t((p->K + L::kScores - 1) / L::kScores));
  gnm_t8_narrow<NMT, NS><<<grid, kT8NrThreads, L::kTotal, s>>>(
      t->nmap8_dos, t->nmap8_mis, pmap, a);
  check_cuda(cudaGetLastError(), "narrow 8-bit tensor launch");
}

// People tiles of 256 instead of 512 when the slowest CTA's share of 512-person
// tiles holds over 1.25 times the work of its share of 256-person tiles (a last
// tile that is mostly padding, a cohort of a few hundred people).  Otherwise
// 512: half the limb traffic per person.  100,000 variants x 16 scores,
// 20,000 people: 191 us on 512-person tiles, 266 us on 256-person ones; 10,000
// variants: 44 and 50 us.
static bool narrow_small_tiles(uint32_t ncta, uint64_t people, uint64_t stages) {
  const uint64_t u4 = (people + 511) / 512 * stages, u2 = (people + 255) / 256 * stages;
  const uint64_t q4 = (u4 + ncta - 1) / ncta, q2 = (u2 + ncta - 1) / ncta;
  return 8 * q4 > 5 * q2;
}

void tensor_accumulate(gnm_plan* p, const uint8_t* d_rows, uint64_t pitch, uint64_t v0,
                       uint64_t nv, cudaStream_t s) {
  TensorPlan* t = p->tensor;
  if (v0 % kTcK != 0)
    fail(GNM_ERR_INVALID, "tensor engine blocks must start at a multiple of 64 variants");
  if (people_as_m(p) && v0 % kT8K == 0) {
    T8NrArgs a{};
    a.a_x0 = int32_t(v0);
    a.part_sum = t->d_slot_sum;
    a.part_cnt = t->d_slot_cnt;
    a.P_pad = t->P_nar;
    a.slot_stride = t->nslot;
    a.err = p->d_err;
    a.stages = uint32_t((nv + kT8K - 1) / kT8K);
    a.state = t->d_state;
    a.quanta = t->d_quanta8;
    a.K_pad = t->K_pad;
    a.K16 = (p->K + kNrScores - 1) / kNrScores * kNrScores;
    if (t->nscores == 2)
      launch_t8_narrow<2, 2>(p, d_rows, pitch, nv, a, s);
    else if (narrow_small_tiles(narrow_ctas(t, p->K, 1), p->fam, a.stages))
      launch_t8_narrow<2, 1>(p, d_rows, pitch, nv, a, s);
    else
      launch_t8_narrow<4, 1>(p, d_rows, pitch, nv, a, s);
    t->slots_used = true;
    p->launches += 1;
    return;
  }
  if (t->narrow) {
    const CUtensorMap pmap = make_row_map(d_rows, p->bpv, nv, pitch, kNrM / 4, kTcK);
    check_cuda(raise_smem_limit(reinterpret_cast<const void*>(gnm_tc_narrow), int(NrSmem::kTotal)),
               "narrow shared memory");
    NrArgs a;
    a.num_rows = nv;
    a.a_x0 = int32_t(v0);
    const uint32_t nall = uint32_t((nv + kTcK - 1) / kTcK);
    a.stages_per_split = (nall + t->nsplits - 1) / t->nsplits;
    a.part_sum = t->d_slot_sum;
    a.part_cnt = t->d_slot_cnt;
    a.P_pad = t->P_nar;
    a.slot_stride = t->nslot;
    a.err = p->d_err;
    gnm_tc_open_slots<<<296, 256, 0, s>>>(t->d_slot_sum, t->d_slot_cnt, t->nslot, t->nsplits,
                                          t->d_state);
    check_cuda(cudaGetLastError(), "narrow slots launch");
    const dim3 grid(uint32_t((p->fam + kNrM - 1) / kNrM),
                    uint32_t((p->K + kNrScores - 1) / kNrScores), t->nsplits);
    gnm_tc_narrow<<<grid, kNrThreads, NrSmem::kTotal, s>>>(t->nmap_dos, t->nmap_mis, pmap, a);
    check_cuda(cudaGetLastError(), "narrow tensor launch");
    p->launches += 2;
    return;
  }
  if (!t->wide_clear) {   // the reset met a plan that runs people as M
    if (t->can_narrow) {
      clear_wide(t, s);
    } else {
      gnm_tc_open_wide<<<296, 256, 0, s>>>(t->d_part_sum, t->d_part_cnt, t->K_pad * t->P_pad,
                                           t->d_state);
      check_cuda(cudaGetLastError(), "wide partials launch");
      p->launches += 1;
    }
  }
  if (t->i8 && v0 % kT8K == 0) {   // a pinned wide shape
    // dosage limbs 0-1 and 2-3, correction limbs 0-1 and 2-3, then the counts
    const CUtensorMap pmap8 = make_row_map(d_rows, p->bpv, nv, pitch, kTcN / 4, kT8K);
    T8Args b;
    b.num_rows = nv;
    b.a_x0 = int32_t(v0);
    b.part_sum = t->d_part_sum;
    b.part_cnt = t->d_part_cnt;
    b.P_pad = t->P_pad;
    b.K_pad = t->K_pad;
    b.quanta = t->d_quanta8;
    b.err = p->d_err;
    b.raster = p->raster;
    if (b.raster && t->ptiles > 65535u) b.raster = 0;  // grid.y limit
    if (t->pair) {
      // SM pairs, one persistent launch: each CTA loads its 128 people's
      // packed bytes (32 per row)
      const CUtensorMap pmap_half = make_row_map(d_rows, p->bpv, nv, pitch, kTcN / 8, kT8K);
      T8PairArgs c;
      c.num_rows = nv;
      c.a_x0 = int32_t(v0);
      c.part_sum = t->d_part_sum;
      c.part_pass = t->d_part_pass;
      c.part_cnt = t->d_part_cnt;
      c.P_pad = t->P_pad;
      c.K_pad = t->K_pad;
      c.quanta = t->d_quanta8;
      c.err = p->d_err;
      c.raster = p->raster;
      c.ptiles = t->ptiles;
      c.spairs = (t->stiles + 1) / 2;
      c.spairs_m = (c.spairs + 1) / 2;
      c.items = 4 * c.ptiles * c.spairs + c.ptiles * c.spairs_m;
      c.store = t->pass_valid ? 0u : 1u;
      launch_t8_pairs(t->map8_2, t->map8_1, pmap_half, c, p->device, s);
      t->pass_valid = true;
      p->launches += 1;
      return;
    }
    for (int32_t z : {0, 2}) {
      b.z0 = z;
      check_cuda((launch_t8<2, kT8StagesPair, false, false>(t->map8_2, pmap8, b, t->ptiles,
                                                        t->stiles, s)),
                 "8-bit tensor dosage launch");
    }
    for (int32_t z : {4, 6}) {
      b.z0 = z;
      check_cuda((launch_t8<2, kT8StagesPair, true, false>(t->map8_2, pmap8, b, t->ptiles,
                                                       t->stiles, s)),
                 "8-bit tensor missing launch");
    }
    b.z0 = 8;
    check_cuda((launch_t8<1, kT8StagesOne, true, true>(t->map8_1, pmap8, b, t->ptiles, t->stiles,
                                                    s)),
               "8-bit tensor count launch");
    p->launches += 5;
    return;
  }
  const CUtensorMap pmap = make_row_map(d_rows, p->bpv, nv, pitch, kTcN / 4, kTcK);
  TcArgs a;
  a.num_rows = nv;
  a.a_x0 = int32_t(v0);
  a.part_sum = t->d_part_sum;
  a.part_cnt = t->d_part_cnt;
  a.P_pad = t->P_pad;
  a.err = p->d_err;
  a.raster = p->raster;
  if (a.raster && t->ptiles > 65535u) a.raster = 0;  // grid.y limit
  // dosage limbs 0-1 and 2-3, then correction limbs 0-1 and (limb 2, count)
  a.z0 = 0;
  check_cuda((launch_tc<kTcPlanes, kTcStages, false, false>(t->map_dos, pmap, a, t->ptiles,
                                                            t->stiles, s)),
             "tensor dosage launch");
  a.z0 = 2;
  check_cuda((launch_tc<kTcPlanes, kTcStages, false, false>(t->map_dos, pmap, a, t->ptiles,
                                                            t->stiles, s)),
             "tensor dosage launch");
  a.z0 = 0;
  check_cuda((launch_tc<kTcPlanes, kTcStages, true, false>(t->map_mis, pmap, a, t->ptiles,
                                                           t->stiles, s)),
             "tensor missing launch");
  a.z0 = 2;
  check_cuda((launch_tc<kTcPlanes, kTcStages, true, true>(t->map_mis, pmap, a, t->ptiles,
                                                          t->stiles, s)),
             "tensor missing launch");
  p->launches += 4;
}

void tensor_finalize(gnm_plan* p, double* d_sums, uint32_t* d_counts, bool add_baseline,
                     cudaStream_t s) {
  TensorPlan* t = p->tensor;
  const uint64_t n = p->P * p->K;
  if (n == 0) return;
  const double* init = add_baseline ? p->d_baseline : p->d_zero_base;
  const uint32_t gx = uint32_t((p->P + 31) / 32);
  // over 64 scores, blocks that ran a wide kernel lie in the wide partials
  const bool slots = t->narrow || t->slots_used || people_as_m(p);
  const bool wide = t->can_narrow ? t->wide_clear && !slots : true;
  const SlotSums ss{slots ? t->d_slot_sum : nullptr, t->d_slot_cnt, t->P_nar, t->nslot,
                    t->d_state};
  const WideSums ws{wide ? t->d_part_sum : nullptr, t->d_part_cnt,
                    t->pass_valid ? t->d_part_pass : nullptr, t->P_pad, t->K_pad * t->P_pad,
                    t->wide_clear ? nullptr : t->d_state + 2};
  // Many slots (few people tiles) are summed by more warps per output: 1,503 people x
  // 30,011 variants x 12, 30 against 41 us for the whole call; four or fewer leave
  // the 32 x 32 blocks ahead (100,000 x 4,000 x 16: 69 against 81 us; x 512: 1.49
  // against 1.88 ms).
  const bool many = slots && t->nslots8 > 4;
  const uint32_t per = many ? kSlotScores : kFinTile;
  const uint32_t ktiles = uint32_t((p->K + per - 1) / per);
  for (uint32_t y = 0; y < ktiles; y += kGridY) {   // a grid has at most 65,535 rows
    const dim3 grid(gx, std::min(kGridY, ktiles - y));
    if (many)
      gnm_tc_finalize_slots<<<grid, 32 * kSlotWarps, 0, s>>>(ss, ws, init, p->d_out_to_fam, p->P,
                                                             p->K, y, d_sums, d_counts);
    else
      gnm_tc_finalize<<<grid, 256, 0, s>>>(ss, ws, init, p->d_out_to_fam, p->P, p->K, y, d_sums,
                                           d_counts);
    check_cuda(cudaGetLastError(), "tensor finalize launch");
    p->launches += 1;
  }
}

static void launch_bw_amax(const gnm_plan* p, const float* gsf, uint32_t* amax, BwSpread spread,
                           cudaStream_t s) {
  const uint64_t n = p->fam * p->K;
  if (!n) return;
  // 2,048 values per CTA, more where that would be over 2,048 CTAs (each ends with
  // up to 256 x 3 atomics); the shared sums of exponents hold 2^23 rows
  const uint64_t cols = std::min<uint64_t>(256, p->K), height = 256 / cols;
  const uint64_t tiles = (p->K + 255) / 256, steps = (p->fam + 8 * height - 1) / (8 * height);
  const uint64_t most = std::max<uint64_t>(1, 2048 / tiles);
  const uint64_t per = std::min<uint64_t>(uint64_t(1) << 23, (steps + most - 1) / most * 8 * height);
  const dim3 grid(uint32_t((p->fam + per - 1) / per), uint32_t(tiles));
  gnm_bw_amax<<<grid, 256, 0, s>>>(gsf, p->fam, p->K, uint32_t(per), amax, spread);
  check_cuda(cudaGetLastError(), "gradient maximum launch");
}

// dS limbs in 8 bits (gnm_t8_backward): buffers [limb rows][P_pad] int8, [4][K16]
// FP64 quanta, [K16] maxima, segment slots, re-derived on every call.
static void backward_dw8(gnm_plan* p, const uint8_t* d_rows, uint64_t pitch, const float* gsf,
                         float* d_grad_w, float* d_grad_corr, cudaStream_t s) {
  const uint64_t K16 = (p->K + kBwScores - 1) / kBwScores * kBwScores;
  const uint64_t P_pad = std::max<uint64_t>(kBw8K, (p->fam + kBw8K - 1) / kBw8K * kBw8K);
  const uint64_t limb_rows = K16 / kBwScores * kBwN;
  int sms = 0;
  check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p->device),
             "cudaDeviceGetAttribute");
  Bw8Args a;
  a.V = p->V;
  a.K = p->K;
  a.K16 = K16;
  a.stages = uint32_t(P_pad / kBw8K);
  a.vtiles = uint32_t((p->V + kBw8Tile - 1) / kBw8Tile);
  const uint64_t units = uint64_t(a.vtiles) * a.stages, stiles = K16 / kBwScores;
  const uint64_t share = std::max<uint64_t>(1, uint64_t(std::max(1, sms)) / stiles);
  a.quota = uint32_t((units + share - 1) / share);
  // whole tiles per share when that lengthens the longest share by no more than
  // the join costs (about 5 us, four stages of 1.2 us)
  const uint32_t whole = (a.quota + a.stages - 1) / a.stages * a.stages;
  if (whole - a.quota <= 4) a.quota = whole;
  const uint32_t ctas = uint32_t((units + a.quota - 1) / a.quota);

  const uint64_t planes_bytes = (limb_rows * P_pad + 255) / 256 * 256;
  const uint64_t q_bytes = 4 * K16 * 8;
  // per score: exponent sum (8 bytes), maximum, count of non-zero values, `sparse`
  const uint64_t amax_bytes = (K16 * 20 + 255) / 256 * 256;
  const uint64_t part_bytes = 2 * ctas * stiles * kBw8SlotElems * 8;
  const uint64_t need = planes_bytes + q_bytes + amax_bytes + part_bytes;
  if (p->bw_bytes < need) {
    check_cuda(cudaStreamSynchronize(s), "backward buffer resize");
    pool_free(p->d_bw);
    p->d_bw = nullptr;
    p->device_bytes -= p->bw_bytes;
    p->bw_bytes = 0;
    p->d_bw = static_cast<uint8_t*>(pool_alloc(p->device, need, "backward dS limbs"));
    p->bw_bytes = need;
    p->device_bytes += need;
  }
  auto* planes = reinterpret_cast<int8_t*>(p->d_bw);
  auto* quanta = reinterpret_cast<double*>(p->d_bw + planes_bytes);
  auto* exps = reinterpret_cast<unsigned long long*>(p->d_bw + planes_bytes + q_bytes);
  auto* amax = reinterpret_cast<uint32_t*>(exps + K16);
  const BwSpread spread{exps, amax + K16};
  auto* sparse = amax + 2 * K16;
  a.quanta = quanta;
  a.sparse = sparse;
  a.part = reinterpret_cast<double*>(p->d_bw + planes_bytes + q_bytes + amax_bytes);
  a.gw = d_grad_w;
  a.gc = d_grad_corr;
  a.err = p->d_err;
  a.rows = d_rows;
  a.pitch = pitch;
  a.ds = gsf;
  a.people = p->fam;
  check_cuda(cudaMemsetAsync(exps, 0, K16 * 16, s), "memset");
  launch_bw_amax(p, gsf, amax, d_grad_corr ? spread : BwSpread{}, s);
  gnm_bw_build8<<<dim3(uint32_t(P_pad / 32), uint32_t(stiles)), 512, 0, s>>>(
      gsf, p->fam, p->K, K16, P_pad, amax, spread, planes, quanta, sparse);
  check_cuda(cudaGetLastError(), "gradient limb launch");

  const CUtensorMap rmap = make_row_map(d_rows, p->bpv, p->V, pitch, Bw8Smem::kPkRow, kBw8Tile,
                                        CU_TENSOR_MAP_SWIZZLE_128B);
  const CUtensorMap bmap =
      make_2d_map(CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, planes, P_pad, limb_rows, 128, kBwN,
                  CU_TENSOR_MAP_SWIZZLE_128B, "gradient limbs");
  const dim3 grid(ctas, uint32_t(stiles));
  auto launch = [&](auto kernel) {
    check_cuda(raise_smem_limit(reinterpret_cast<const void*>(kernel), int(Bw8Smem::kTotal)),
               "backward shared memory");
    kernel<<<grid, kBw8Threads, Bw8Smem::kTotal, s>>>(rmap, bmap, a);
    check_cuda(cudaGetLastError(), "backward launch");
  };
  if (d_grad_corr)
    launch(gnm_t8_backward<true>);
  else
    launch(gnm_t8_backward<false>);
  p->launches += 3;
  if (a.quota % a.stages != 0 && ctas > 1) {   // some tile spans shares
    gnm_bw_join<<<dim3(ctas - 1, uint32_t(stiles), 8), 256, 0, s>>>(a, ctas);
    check_cuda(cudaGetLastError(), "backward join launch");
    p->launches += 1;
  }
}

void backward_dw(gnm_plan* p, const uint8_t* d_rows, uint64_t pitch, const float* d_grad_s,
                 float* d_grad_w, float* d_grad_corr, cudaStream_t s) {
  if (!d_rows || !d_grad_s || !d_grad_w) fail(GNM_ERR_INVALID, "NULL buffer");
  if (pitch < p->bpv) fail(GNM_ERR_INVALID, "pitch smaller than bytes per variant");
  if (pitch % 16 != 0 || reinterpret_cast<uintptr_t>(d_rows) % 16 != 0)
    fail(GNM_ERR_INVALID, "packed rows must be 16-byte aligned with a pitch multiple of 16");
  if (p->V == 0) return;
  const float* gsf = d_grad_s;
  if (p->d_out_to_fam || p->P != p->fam) {
    // dS rows in .bed person order: zero for people outside the keep set
    if (!p->d_grad_fam) {
      p->d_grad_fam = static_cast<float*>(
          pool_alloc(p->device, std::max<uint64_t>(1, p->fam * p->K) * 4, "fam-order gradient"));
      p->device_bytes += p->fam * p->K * 4;
    }
    check_cuda(cudaMemsetAsync(p->d_grad_fam, 0, p->fam * p->K * 4, s), "memset");
    const uint64_t n = p->P * p->K;
    if (n) {
      gnm_scatter_grad<<<uint32_t((n + 255) / 256), 256, 0, s>>>(
          d_grad_s, p->d_out_to_fam, p->P, p->K, p->d_grad_fam);
      check_cuda(cudaGetLastError(), "gradient scatter launch");
      p->launches += 1;
    }
    gsf = p->d_grad_fam;
  }
  if (p->bw_limb_bits == 8) {
    backward_dw8(p, d_rows, pitch, gsf, d_grad_w, d_grad_corr, s);
    return;
  }
  // dS limb rows and the FP32 copy, re-derived on every call
  const uint64_t K16 = (p->K + kBwScores - 1) / kBwScores * kBwScores;
  const uint64_t P_pad = std::max<uint64_t>(kBwK, (p->fam + kBwK - 1) / kBwK * kBwK);
  const uint64_t limb_rows = K16 / kBwScores * kBwN;
  const uint64_t planes_bytes = (limb_rows * P_pad * 2 + 255) / 256 * 256;
  const uint64_t ds_bytes = (P_pad * K16 * 4 + 255) / 256 * 256;
  const uint64_t need = planes_bytes + ds_bytes + K16 * 4;
  if (p->bw_bytes < need) {
    check_cuda(cudaStreamSynchronize(s), "backward buffer resize");
    pool_free(p->d_bw);
    p->d_bw = nullptr;
    p->device_bytes -= p->bw_bytes;
    p->bw_bytes = 0;
    p->d_bw = static_cast<uint8_t*>(pool_alloc(p->device, need, "backward dS limbs"));
    p->bw_bytes = need;
    p->device_bytes += need;
  }
  auto* planes = reinterpret_cast<__nv_bfloat16*>(p->d_bw);
  auto* ds = reinterpret_cast<float*>(p->d_bw + planes_bytes);
  auto* amax = reinterpret_cast<uint32_t*>(p->d_bw + planes_bytes + ds_bytes);
  check_cuda(cudaMemsetAsync(amax, 0, K16 * 4, s), "memset");
  launch_bw_amax(p, gsf, amax, BwSpread{}, s);
  p->launches += 1;
  const uint64_t nb = K16 * P_pad;
  gnm_bw_build<<<uint32_t((nb + 255) / 256), 256, 0, s>>>(gsf, p->fam, p->K, K16, P_pad, amax,
                                                          planes, ds);
  check_cuda(cudaGetLastError(), "gradient limb launch");
  p->launches += 1;

  const CUtensorMap rmap = make_row_map(d_rows, p->bpv, p->V, pitch, kBwK / 4, kBwM);
  const CUtensorMap bmap =
      make_2d_map(CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, planes, P_pad, limb_rows, kBwK, kBwN,
                  CU_TENSOR_MAP_SWIZZLE_128B, "gradient limbs");
  const CUtensorMap dmap = make_2d_map(CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, ds, K16, P_pad,
                                       kBwScores, kBwK, CU_TENSOR_MAP_SWIZZLE_NONE, "gradient");
  check_cuda(raise_smem_limit(reinterpret_cast<const void*>(gnm_tc_backward), int(BwSmem::kTotal)),
             "backward shared memory");
  BwArgs a;
  a.V = p->V;
  a.K = p->K;
  a.nstages = uint32_t(P_pad / kBwK);
  a.gw = d_grad_w;
  a.gc = d_grad_corr;
  a.err = p->d_err;
  const dim3 grid(uint32_t((p->V + kBwM - 1) / kBwM), uint32_t(K16 / kBwScores));
  gnm_tc_backward<<<grid, kBwThreads, BwSmem::kTotal, s>>>(rmap, bmap, dmap, a);
  check_cuda(cudaGetLastError(), "backward launch");
  p->launches += 1;
}

}  // namespace gnm
