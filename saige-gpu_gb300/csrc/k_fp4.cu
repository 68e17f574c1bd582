// Exact-integer genotype GEMMs on the FP4 tensor pipe (tcgen05 kind::mxf4), sm_103a.
//
//   D[j, r] = 2^-e_j sum_k G[r, k] q_j[k],   G in {0, 1, 2},  |q_j| <= 2^24 integers
//
// G is exact in E2M1.  A vector enters as a fixed-point column q_j = rint(2^e_j v_j), its largest
// magnitude brought into (2^23, 2^24], and each q as seven base-13 digits.  The digit set
// {0, +-1, +-2, +-3, +-4, +-6, +-8} holds one representative of every residue mod 13 and every one
// of them is (twice) an E2M1 value, so a digit is one FP4 element: 3.7 bits of the vector per FP4
// element against 8 per BF16 element, on a pipe with six times the rate.  Seven digits cover
// |q| <= 20,544,880.
//
// Every digit has its own FP32 accumulator in TMEM.  A product is at most 16 in units of 1/2, so
// sums over up to 2^20 elements of K are integers below 2^24: the accumulation is exact, needs no
// draining, and cannot depend on tiling.  The epilogue combines the seven sums in 64-bit integers
// and rounds once, to FP32: the only errors of a product are the quantisation of v (2^-25 of the
// column's largest entry, against 2^-17 of each entry for BF16 high + low halves) and that rounding.
// Reductions longer than 2^20 run in segments, added in FP32.
//
// Layout.  Both operands are stored as the MMA reads them from shared memory (K-major, no swizzle:
// core matrices of 8 rows x 16 bytes), one K stage of 192 elements at a time: [8-row group][6 chunks
// of 32 elements][8 rows][16 bytes].  A (row block, stage) of G is then 12,288 contiguous bytes, and
// so is a CTA's share of a column tile, so a stage is two long contiguous TMA reads: G streams from
// HBM at the copy rate however far apart its rows are.  192 = 2 x 96 elements: the K = 96 form of
// the MMA (sm_103a) runs 1.5 times the rate of K = 64 (measured 24,574 against 16,383 MAC per clock
// and SM).
//
// What runs here: the subset-exact products of the drop-ins that return FP32 (few columns, so G's
// stream from HBM bounds them: half a byte a genotype and product against two).  Measured at N = 100k,
// M = 150k, both products and the kernels around them: 15.0 against 62.2 ms for one AI score (4.1x); the
// 32-column GEMM 1.08 ms, 7.5 GB at 1.02 of the copy rate.
//
// CTA pairs (cta_group::2): a pair computes 256 rows x CT vector columns (7 CT accumulator columns,
// 448 of the 512 TMEM columns at CT = 64).  Block scales are 1.0 (E8M0 127) in 32 TMEM columns
// filled once per CTA.
#include "sg_internal.h"
#include "tc_common.cuh"
#include "geno_bits.cuh"

#include <algorithm>
#include <cmath>

namespace sg {

namespace {

using namespace tc;

constexpr int kDigits = 7;
constexpr int kStageK = kFp4StageK;                 // 192 elements of K per stage
constexpr int kRowStage = kStageK / 2;              // 96 bytes of one row per stage
constexpr int kGroupStage = 8 * kRowStage;          // 768 bytes of an 8-row group per stage
constexpr int kAStage = 128 * kRowStage;            // 12,288 bytes of a row block per stage
constexpr int kSegStages = (1 << 20) / kStageK;     // stages whose digit sums stay below 2^24
constexpr int kMapRow = 256;                        // the TMA maps see the operands as rows of 256 bytes

constexpr int kEpiWarps = 8;
constexpr int kProducerWarp4 = 8;
constexpr int kMmaWarp4 = 9;
constexpr int kFp4Threads = 320;

// E2M1 code of the digit that represents residue r mod 13 (nibble r), and the residues whose digit
// is negative (a carry of one into the next digit).
constexpr uint64_t kDigitCodes = 0x9ABC6D5E43210ull;
constexpr uint32_t kDigitCarry = 0x1EA0u;
constexpr uint32_t kDigitBias = 62748517u;  // 13^7: makes q non-negative without changing a digit
constexpr uint32_t kDiv13 = 330382100u;     // ceil(2^32 / 13): exact quotients below 2^30

// seven E2M1 digit codes of q, lowest digit first, in the low 28 bits
__host__ __device__ __forceinline__ uint32_t digit_codes(int32_t q) {
  uint32_t x = (uint32_t)q + kDigitBias, w = 0;
#pragma unroll
  for (int d = 0; d < kDigits; ++d) {
    const uint32_t t = (uint32_t)(((uint64_t)x * kDiv13) >> 32);
    const uint32_t r = x - 13u * t;
    w |= ((uint32_t)(kDigitCodes >> (4u * r)) & 15u) << (4 * d);
    x = t + ((kDigitCarry >> r) & 1u);
  }
  return w;
}

// Exponent of the power of two that brings a column of magnitude at most ``bound`` into (2^23, 2^24] (exact), and 0
// for a zero column; clamped where its inverse, the descale, would leave FP32 (it may be a subnormal).
__device__ __forceinline__ int fixed_exponent(float bound) {
  if (!(bound > 0.0f)) return 0;
  int e = 0;
  frexpf(bound, &e);  // bound = f 2^e, f in [0.5, 1)
  return min(max(24 - e, -120), 148);
}

// x 2^e in two factors, each within FP32: 2^e alone leaves it for columns below 2^-103
struct Scale {
  float a, b;
  __device__ __forceinline__ explicit Scale(int e) : a(ldexpf(1.0f, e / 2)), b(ldexpf(1.0f, e - e / 2)) {}
  __device__ __forceinline__ float operator()(float x) const { return x * a * b; }
};

// Byte of vector column j's digit d, element k, in the digit operand of column tiles of CT columns
// (S stages): tile, stage and CTA rank of the pair, then the CTA's rows (half h of 32 columns has
// 224 rows, or 112 where only 16 columns are left; each rank holds half of a half's rows).
struct DigitTile {
  int32_t ct, stages;
};
struct DigitColumn {
  int64_t base;  // the column tile's first byte
  int h, r, hn;  // half, first row within it, rows of it that each rank holds
};
__device__ __forceinline__ DigitColumn digit_column(const DigitTile t, int j) {
  const int tile = j / t.ct, c = j - tile * t.ct, h = c >> 5;
  return DigitColumn{(int64_t)tile * t.stages * (672 * (int64_t)t.ct), h, (c & 31) * kDigits,
                     t.ct - 32 * h >= 32 ? 112 : 56};
}

// No-swizzle K-major descriptor: 128 bytes between core matrices along K, 768 between 8-row groups.
__device__ __forceinline__ uint64_t smem_desc_fp4(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(128 >> 4) << 16;
  d |= (uint64_t)(kGroupStage >> 4) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// Instruction descriptor of kind::mxf4: E2M1 operands (1), E8M0 scales (bit 23), N >> 3 at bit 17,
// M >> 4 at bit 24, K = 96 (bit 31).
__host__ __device__ constexpr uint32_t fp4_idesc(int n) {
  return (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | ((uint32_t)(256 >> 4) << 24) | (1u << 31);
}

__device__ __forceinline__ void umma_fp4(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa,
                                         uint32_t sfb, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %6, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.block32 [%0], %1, %2, %3, [%4], [%5], p;\n\t}"
      ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accumulate));
}

// 56 consecutive TMEM columns (eight vector columns of seven digits) of this warp's 32 lanes
__device__ __forceinline__ void tmem_ld56(uint32_t taddr, uint32_t (&r)[56]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47])
      : "r"(taddr + 32));
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55])
               : "r"(taddr + 48));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// What a tile's sums become: D = FP32 of sum x descale (kProduct); the 64-bit sums themselves (kSums); the
// GRM's entries (kSyrk, see fp4_syrk).
enum { kProduct = 0, kSums = 1, kSyrk = 2 };

// kSyrk: tiles come from a table (row block, column tile), and entry (r, c), c <= r < n, is
// (sum - shift[r] - shift[c] + c0) scale, written to K[r][c] and K[c][r] (rows past n: zero).
struct SyrkArgs {
  const int2* tiles;
  const long long* shift;
  long long c0;
  float scale;
  int64_t n;
};

// The sum of seven digits' accumulators: integers below 2^24 in units of 1/2.  ``magic``: below 2^22,
// where adding 1.5 2^23 leaves the integer in the low mantissa bits (a conversion takes a quarter-rate
// instruction).
__device__ __forceinline__ long long combine_digits(const uint32_t* v, bool magic) {
  long long t = 0;
#pragma unroll
  for (int d = kDigits - 1; d >= 0; --d) {
    const float x = __uint_as_float(v[d]);
    const int s = magic ? (__float_as_int(fmaf(x, 2.0f, 12582912.0f)) - 0x4B400000) : __float2int_rn(2.0f * x);
    t = 13 * t + s;
  }
  return t;
}

// One 256-row x CT-column tile per CTA pair.  Warp 8 (one lane) loads a stage's rows of G and of the
// digits into an S-stage ring (the pair's loads complete on the leader's barrier); warp 9 of the
// leader issues two K = 96 MMAs per stage and 32-column half; warps 0-7 combine and store.
// Tiles run column tiles fastest, so the pairs resident at one time share their strips of G in L2.
template <int CT, int S, int kMode>
__global__ void __launch_bounds__(kFp4Threads, CT <= 32 ? 2 : 1)
fp4_gemm_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, int stages,
                int ncolt, void* __restrict__ Dv, int64_t ldd, int64_t nrows, const float* __restrict__ descale,
                const SyrkArgs sy, int* __restrict__ err) {
  constexpr int kHalves = CT > 32 ? 2 : 1;
  constexpr int kN0 = CT >= 32 ? 224 : 112, kN1 = CT == 64 ? 224 : 112;
  constexpr int kBStage = 336 * CT;               // this CTA's digit rows (3.5 CT) per stage
  constexpr int kStage = kAStage + kBStage;
  constexpr uint32_t kSfCol = kHalves == 2 ? 448 : 224;  // 32 TMEM columns of unit block scales
  constexpr uint32_t kTmem = kHalves == 2 ? 512 : 256;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + S * kStage);
  uint64_t* empty = full + S;
  uint64_t* acc_full = empty + S;    // a segment's MMAs have completed
  uint64_t* acc_empty = acc_full + 1;  // the epilogue warps of both CTAs have read it
  uint64_t* mma_done = acc_empty + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mma_done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t crank = cluster_rank();
  const bool leader = crank == 0;
  const int tile = blockIdx.x >> 1;
  int rt, bt;
  if constexpr (kMode == kSyrk) {
    const int2 tc = sy.tiles[tile];
    rt = tc.x;
    bt = tc.y;
  } else {
    rt = tile / ncolt;
    bt = tile - rt * ncolt;
  }
  const int row_block = 2 * rt + (int)crank;

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    mbar_init(acc_empty, 2 * kEpiWarps);
    mbar_init(mma_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == kMmaWarp4) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmem)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  if (warp < 4) {  // unit scales in every lane
    const uint32_t one = 0x7F7F7F7Fu;
#pragma unroll
    for (int c = 0; c < 32; ++c)
      asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};"
                   ::"r"(tmem + ((uint32_t)(warp * 32) << 16) + kSfCol + (uint32_t)c), "r"(one) : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();  // both CTAs' barriers and scales exist before either signals the other
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  if (warp == kProducerWarp4) {
    if (elect_one()) {
      const int64_t ra = (int64_t)row_block * stages, rb = (int64_t)bt * stages * 2 + crank;
      int issued = 0;
      for (int kb = 0; kb < stages; ++kb) {
        const int s = kb % S;
        if (!mbar_wait(&empty[s], ((uint32_t)(kb / S) & 1u) ^ 1u, 1, abort_flag, err)) break;
        uint8_t* st = smem + s * kStage;
        const uint32_t fb = cluster_addr(&full[s], 0);
        if (leader) mbar_expect_tx(&full[s], 2u * (uint32_t)kStage);
        tma_load_2d_pair(st, &mapA, fb, 0, (int32_t)((ra + kb) * (kAStage / kMapRow)));
        tma_load_2d_pair(st + kAStage, &mapB, fb, 0, (int32_t)((rb + 2 * kb) * (kBStage / kMapRow)));
        issued = kb + 1;
      }
      // after an abort: the loads in flight land before the shared memory is given up
      if (*abort_flag && leader)
        for (int kb = issued > S ? issued - S : 0; kb < issued; ++kb)
          mbar_wait_teardown(&full[kb % S], (uint32_t)(kb / S) & 1u);
    }
  } else if (warp == kMmaWarp4) {
    if (leader && elect_one()) {
      const uint32_t empty_peer = cluster_addr(empty, 1), accf_peer = cluster_addr(acc_full, 1);
      int kb = 0;
      bool go = true;
      for (int seg = 0; go && kb < stages; ++seg) {
        const int end = stages - kb < kSegStages ? stages : kb + kSegStages;
        if (seg > 0) {
          go = mbar_wait(acc_empty, (uint32_t)(seg - 1) & 1u, 5, abort_flag, err);
          if (!go) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        const int first = kb;
        for (; kb < end; ++kb) {
          const int s = kb % S;
          if (!mbar_wait(&full[s], (uint32_t)(kb / S) & 1u, 2, abort_flag, err)) {
            go = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a0 = smem_u32(smem + s * kStage), b0 = a0 + kAStage;
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const uint32_t acc = (kb > first || k > 0) ? 1u : 0u;
            const uint64_t da = smem_desc_fp4(a0 + 384u * k);
            umma_fp4(tmem, da, smem_desc_fp4(b0 + 384u * k), fp4_idesc(kN0), tmem + kSfCol, tmem + kSfCol + 16, acc);
            if constexpr (kHalves == 2)  // the second half's rows follow the first's 112
              umma_fp4(tmem + 224, da, smem_desc_fp4(b0 + 14 * kGroupStage + 384u * k), fp4_idesc(kN1), tmem + kSfCol,
                       tmem + kSfCol + 16, acc);
          }
          umma_commit<true>(smem_u32(&empty[s]));
          umma_commit<true>(empty_peer + (uint32_t)s * 8u);
        }
        if (go) {
          umma_commit<true>(smem_u32(acc_full));
          umma_commit<true>(accf_peer);
        }
      }
      umma_commit<true>(smem_u32(mma_done));
      mbar_wait_teardown(mma_done, 0u);
    }
  } else {
    const int quad = warp & 3, half = warp >> 2;
    const uint32_t tl = tmem + ((uint32_t)(quad * 32) << 16);
    const int64_t r = (int64_t)row_block * 128 + quad * 32 + lane;
    const uint32_t acce_leader = cluster_addr(acc_empty, 0);
    const int nseg = (stages + kSegStages - 1) / kSegStages;
    const bool magic = stages <= (1 << 22) / (16 * kStageK);
    for (int seg = 0; seg < nseg; ++seg) {
      int go = 1;
      if (lane == 0) go = mbar_wait_sleep(acc_full, (uint32_t)seg & 1u, 3, abort_flag, err) && !*abort_flag;
      go = __shfl_sync(0xffffffffu, go, 0);
      __syncwarp();
      if (!go) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int b = half; b < CT / 8; b += 2) {
        uint32_t v[56];
        tmem_ld56(tl + (uint32_t)(56 * b), v);
        if ((int64_t)row_block * 128 >= nrows) continue;
        const int64_t j0 = (int64_t)bt * CT + 8 * b;
        if constexpr (kMode == kProduct) {
          float* D = static_cast<float*>(Dv);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float x = __ll2float_rn(combine_digits(v + 7 * c, magic)) * __ldg(descale + j0 + c);
            float* o = D + (j0 + c) * ldd + r;
            *o = seg == 0 ? x : *o + x;
          }
        } else if constexpr (kMode == kSums) {
          long long* D = static_cast<long long*>(Dv);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const long long t = combine_digits(v + 7 * c, magic);
            long long* o = D + (j0 + c) * ldd + r;
            *o = seg == 0 ? t : *o + t;
          }
        } else {  // one segment only (fp4_syrk checks)
          float* K = static_cast<float*>(Dv);
          const long long ar = r < sy.n ? sy.shift[r] : 0;
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const int64_t cc = j0 + c;
            if (cc <= r && cc < nrows) {
              const long long t = combine_digits(v + 7 * c, magic) - ar - __ldg(sy.shift + (cc < sy.n ? cc : 0)) + sy.c0;
              const float x = r < sy.n ? __ll2float_rn(t) * sy.scale : 0.0f;
              K[r * ldd + cc] = x;
              K[cc * ldd + r] = x;
            }
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(acce_leader);
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();  // neither CTA leaves while the other's MMAs or arrivals may still touch it
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == kMmaWarp4)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmem) : "memory");
}

// An operand of ``bytes`` contiguous bytes (a multiple of 256) as rows of 256, boxes of box_rows.
bool fp4_map(CUtensorMap* m, const void* base, int64_t bytes, uint32_t box_rows) {
  auto fn = tc_encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[2] = {kMapRow, (cuuint64_t)(bytes / kMapRow)};
  const cuuint64_t strides[1] = {kMapRow};
  const cuuint32_t box[2] = {kMapRow, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ntiles tiles of 256 rows x CT columns, column tiles (ncolt) fastest.
template <int CT, int S, int kMode>
cudaError_t launch_fp4(const CUtensorMap& a, const CUtensorMap& b, int stages, int64_t rows, int64_t ntiles, int ncolt,
                       void* D, int64_t ldd, const float* descale, const SyrkArgs& sy, int* err, cudaStream_t s) {
  auto k = fp4_gemm_kernel<CT, S, kMode>;
  constexpr size_t sm = (size_t)S * (kAStage + 336 * CT) + 128 + 256;
  static_assert(sm <= 232448 && 2 * S + 4 <= 31, "stage ring and barriers fit the CTA's shared memory");
  cudaError_t e = set_dynamic_smem(reinterpret_cast<const void*>(k), sm);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * ntiles));
  cfg.blockDim = dim3(kFp4Threads);
  cfg.dynamicSmemBytes = sm;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, k, a, b, stages, ncolt, D, ldd, rows, descale, sy, err);
  return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace

// ----------------------------------------------------------------------------------- genotypes
// G in E2M1 (0, 1, 2 -> codes 0, 2, 4) from the packed codes, 16 at a time: a word of codes becomes a word of copies
// (pack_copies), and that two words of E2M1.  Missing calls take the cohort fill (no fill: there are none); rows and
// elements past the ends are zero.  Both builds write 16 contiguous bytes a thread; bound by that and by the integer
// work on the words.  At N = 100,000, M = 150,000 (15 GB written): the rows of markers from 10.0 to 2.5 ms, the rows of
// samples from 13.7 to 7.0 (a code at a time before).

// fields 0..7 of two bits to the low halves of nibbles 0..7
__device__ __forceinline__ uint32_t spread_nibbles(uint32_t x) {
  x = (x | (x << 8)) & 0x00FF00FFu;
  x = (x | (x << 4)) & 0x0F0F0F0Fu;
  return (x | (x << 2)) & 0x33333333u;
}
__device__ __forceinline__ uint2 fp4_of_copies(uint32_t w) {
  return make_uint2(spread_nibbles(w & 0xFFFFu) << 1, spread_nibbles(w >> 16) << 1);
}

// Rows of markers: block = (row block of 128 markers, kMmStages stages), 16 bytes of codes (64 samples) a thread, turned
// in shared memory and written as whole stages.
constexpr int kMmStages = 4;
constexpr int kMmChunks = 6 * kMmStages;  // chunks of 32 samples of a row
constexpr size_t kMmSmem = (size_t)kMmChunks * 129 * 16;

__global__ void __launch_bounds__(256)
fp4_gbuild_mm_kernel(const uint8_t* __restrict__ codes, int64_t pitch, const int32_t* __restrict__ fill, int64_t m,
                     int64_t nn, int stages, int64_t rows_blocks, uint4* __restrict__ out) {
  extern __shared__ uint4 sp[];  // [chunk][128 rows + 1]
  const int ks0 = blockIdx.x * kMmStages;
  const int64_t rb = blockIdx.y + (int64_t)blockIdx.z * 65535;
  if (rb >= rows_blocks) return;
  for (int t = threadIdx.x; t < 128 * (kMmChunks / 2); t += blockDim.x) {
    const int row = t / (kMmChunks / 2), q = t % (kMmChunks / 2);
    const int64_t mk = rb * 128 + row, s0 = (int64_t)ks0 * kStageK + 64 * q;
    uint2 w[4] = {};
    if (mk < m && s0 < nn) {  // rows are padded to 16 bytes, which is what is read
      const uint4 x = *reinterpret_cast<const uint4*>(codes + mk * pitch + s0 / 4);
      const int f = fill ? fill[mk] : 0;
      const uint32_t c[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = fp4_of_copies(pack_copies(c[i], f, valid_fields(nn - (s0 + 16 * i))));
    }
    sp[(2 * q) * 129 + row] = make_uint4(w[0].x, w[0].y, w[1].x, w[1].y);
    sp[(2 * q + 1) * 129 + row] = make_uint4(w[2].x, w[2].y, w[3].x, w[3].y);
  }
  __syncthreads();
  constexpr int kStageQ = kAStage / 16;
  for (int t = threadIdx.x; t < kMmStages * kStageQ; t += blockDim.x) {
    const int ks = ks0 + t / kStageQ, u = t % kStageQ;
    const int row = (u / 48) * 8 + (u & 7), chunk = (t / kStageQ) * 6 + (u >> 3) % 6;
    if (ks < stages) out[(rb * stages + ks) * kStageQ + u] = sp[chunk * 129 + row];
  }
}

// Rows of samples: block = one stage (192 markers) x 256 samples; a thread turns 16 markers x 16 samples of codes
// in registers.
__global__ void __launch_bounds__(192)
fp4_gbuild_sm_kernel(const uint8_t* __restrict__ codes, int64_t pitch, const int32_t* __restrict__ fill, int64_t m,
                     int64_t nn, int stages, uint4* __restrict__ out) {
  // [32 groups of 8 samples][6 chunks][8 samples][2], 8 bytes each; a pair of groups is padded by one, so that half a
  // warp's stores meet every bank once
  constexpr int kPair = 2 * 6 * 8 * 2 + 1;
  __shared__ uint2 so[16 * kPair];
  const int ks = blockIdx.x, sw = threadIdx.x & 15, mg = threadIdx.x >> 4;
  const int64_t rb0 = 2 * (int64_t)blockIdx.y, s0 = rb0 * 128 + 16 * sw, left = nn - s0;
  const uint32_t valid = valid_fields(left);
  uint32_t w[16];
#pragma unroll
  for (int p = 0; p < 16; ++p) {
    const int64_t mk = (int64_t)ks * kStageK + 16 * mg + p;
    // pitch is a multiple of 16, so a word that starts inside a row ends there
    w[p] = mk < m && left > 0 ? pack_copies(*reinterpret_cast<const uint32_t*>(codes + mk * pitch + s0 / 4),
                                            fill ? fill[mk] : 0, valid)
                              : 0u;
  }
  transpose_fields(w);
#pragma unroll
  for (int i = 0; i < 16; ++i)
    so[sw * kPair + (i >> 3) * 96 + (mg >> 1) * 16 + (i & 7) * 2 + (mg & 1)] = fp4_of_copies(w[i]);
  __syncthreads();
  constexpr int kStageQ = kAStage / 16;
  for (int t = threadIdx.x; t < 2 * kStageQ; t += blockDim.x) {
    const int grp = t / 48, u = t % 48;
    const uint2* p = so + (grp >> 1) * kPair + (grp & 1) * 96 + 2 * u;
    out[((rb0 + t / kStageQ) * stages + ks) * kStageQ + t % kStageQ] = make_uint4(p[0].x, p[0].y, p[1].x, p[1].y);
  }
}

int fp4_stages(int64_t k) { return (int)((k + kStageK - 1) / kStageK); }
int64_t fp4_matrix_bytes(int64_t rows, int64_t k) {
  return (rows + 255) / 256 * 2 * (int64_t)fp4_stages(k) * kAStage;
}
int64_t fp4_digit_bytes(int64_t cols, int64_t k) { return round_up(cols, 64) * (int64_t)fp4_stages(k) * 672; }

static void launch_fp4_gbuild_sm(const uint8_t* codes, int64_t pitch, const int32_t* fill, int64_t m, int64_t nn,
                                 int stages, int64_t row_blocks, void* out, cudaStream_t s) {
  fp4_gbuild_sm_kernel<<<dim3((unsigned)stages, (unsigned)(row_blocks / 2)), 192, 0, s>>>(codes, pitch, fill, m, nn, stages,
                                                                                    static_cast<uint4*>(out));
}

cudaError_t launch_fp4_gbuild(const uint8_t* codes, int64_t pitch, const int32_t* fill, int64_t m, int64_t nn, void* Gmm,
                              void* Gsm, cudaStream_t s) {
  const int64_t m1 = m > 0 ? m : 1;  // a cohort without markers still has its (zero) row blocks
  const int64_t rm = (m1 + 255) / 256 * 2, rs = (nn + 255) / 256 * 2;
  const cudaError_t e = tc::set_dynamic_smem(reinterpret_cast<const void*>(fp4_gbuild_mm_kernel), kMmSmem);
  if (e != cudaSuccess) return e;
  const int sn = fp4_stages(nn);
  dim3 g1((unsigned)((sn + kMmStages - 1) / kMmStages), (unsigned)(rm < 65535 ? rm : 65535),
          (unsigned)((rm + 65534) / 65535));
  fp4_gbuild_mm_kernel<<<g1, 256, kMmSmem, s>>>(codes, pitch, fill, m, nn, sn, rm, static_cast<uint4*>(Gmm));
  launch_fp4_gbuild_sm(codes, pitch, fill, m, nn, fp4_stages(m1), rs, Gsm, s);
  return cudaGetLastError();
}

// ----------------------------------------------------------------------------------- vectors
namespace {

constexpr int kQThreads = 256;
constexpr int kQChunk = 8 * kQThreads;  // elements of a column per block, eight per thread

// Eight consecutive digits-of-q words: digit d's nibbles of the thread's eight elements go to one
// 4-byte word of the operand; the seven words of the digits sit in seven consecutive rows.
__device__ __forceinline__ void store_digits(uint8_t* __restrict__ out, const DigitTile t, int64_t j, int64_t k,
                                             const int32_t (&q)[8]) {
  uint32_t c[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) c[i] = digit_codes(q[i]);
  const int ks = (int)(k / kStageK), kk = (int)(k - (int64_t)ks * kStageK);
  const DigitColumn dc = digit_column(t, (int)j);
  uint8_t* o = out + dc.base + (int64_t)ks * (672 * t.ct) + (kk >> 5) * 128 + ((kk & 31) >> 3) * 4;
#pragma unroll
  for (int d = 0; d < kDigits; ++d) {
    uint32_t w = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) w |= ((c[i] >> (4 * d)) & 15u) << (4 * i);
    const int r = dc.r + d, rank = r >= dc.hn ? 1 : 0, row = 112 * dc.h + r - rank * dc.hn;
    *reinterpret_cast<uint32_t*>(o + rank * (336 * t.ct) + (row >> 3) * kGroupStage + (row & 7) * 16) = w;
  }
}

// The block's sum of v and maximum of m, in thread 0, in a fixed order.
__device__ __forceinline__ void block_sum_max(double& v, float& m, double* sh, float* shm) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    v += __shfl_xor_sync(0xffffffffu, v, o);
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) {
    sh[w] = v;
    shm[w] = m;
  }
  __syncthreads();
  if (threadIdx.x == 0)
    for (int i = 1; i < (int)(blockDim.x >> 5); ++i) {
      v += sh[i];
      m = fmaxf(m, shm[i]);
    }
}

// A column's n block partials combined by the whole block, in a fixed order, into sh[0] and shm[0]
// (the first warp's lanes take every 32nd each; either array may be null).
__device__ __forceinline__ void column_sum_max(const double* __restrict__ part, const float* __restrict__ pmax, int n,
                                               double* sh, float* shm) {
  if (threadIdx.x < 32) {
    double v = 0.0;
    float m = 0.0f;
    for (int b = threadIdx.x; b < n; b += 32) {
      if (part) v += part[b];
      if (pmax) m = fmaxf(m, pmax[b]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      v += __shfl_xor_sync(0xffffffffu, v, o);
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    }
    if (threadIdx.x == 0) {
      sh[0] = v;
      shm[0] = m;
    }
  }
  __syncthreads();
}

}  // namespace

// Block partials of a column's sum over the subset (rows outside it are zero in P) and its largest
// magnitude, kQChunk rows each.
__global__ void __launch_bounds__(kQThreads)
fp4_sums_kernel(const float* __restrict__ Pf, int64_t np, const int32_t* __restrict__ cols, double* __restrict__ part,
                float* __restrict__ pmax, int nblk) {
  __shared__ double sh[kQThreads / 32];
  __shared__ float shm[kQThreads / 32];
  const int64_t j = blockIdx.y;
  const int32_t col = cols[j];
  const int64_t k = (int64_t)blockIdx.x * kQChunk + 8 * threadIdx.x;
  double v = 0.0;
  float mx = 0.0f;
  if (col >= 0 && k < np) {  // np is a multiple of 128: the eight are inside it
    const float4* p = reinterpret_cast<const float4*>(Pf + (int64_t)col * np + k);
    const float4 a = p[0], b = p[1];
    v = (((double)a.x + a.y) + ((double)a.z + a.w)) + (((double)b.x + b.y) + ((double)b.z + b.w));
    mx = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))),
               fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fmaxf(fabsf(b.z), fabsf(b.w))));
  }
  block_sum_max(v, mx, sh, shm);
  if (threadIdx.x == 0) {
    part[j * nblk + blockIdx.x] = v;
    pmax[j * nblk + blockIdx.x] = mx;
  }
}

// v_c = P - mean_S(P) on the subset (0 elsewhere and for padding columns) as base-13 digits; the
// column's mean and descale go to colmean[j] and descale[j], the block sums of the quantised values
// (the mean's rounding times the subset's size) to qsum.  A column that is not finite gets a
// NaN descale, so its product is NaN, as any product with it is.
__global__ void __launch_bounds__(kQThreads)
fp4_center_digits_kernel(const float* __restrict__ Pf, int64_t np, const int32_t* __restrict__ cols,
                         const ColState* __restrict__ st, const SubsetSlot* __restrict__ slots,
                         const double* __restrict__ winv, const double* __restrict__ part,
                         const float* __restrict__ pmax, int nblk, int nsum, DigitTile dt, uint8_t* __restrict__ out,
                         float* __restrict__ colmean, float* __restrict__ descale, double* __restrict__ qsum) {
  __shared__ double sh[kQThreads / 32];
  __shared__ float shm[kQThreads / 32];
  __shared__ float s_mu;
  __shared__ int s_e;
  const int64_t j = blockIdx.y;
  const int32_t col = cols[j];
  const int slot = col >= 0 ? st[col].pheno : 0;
  column_sum_max(part + j * nblk, pmax + j * nblk, col >= 0 ? nsum : 0, sh, shm);
  if (threadIdx.x == 0) {
    const float mu = col >= 0 ? (float)(sh[0] / slots[slot].ns) : 0.0f;
    const float bound = shm[0] + fabsf(mu);  // of |P - mu| over the column
    const int e = fixed_exponent(bound);
    s_mu = mu;
    s_e = e;
    if (blockIdx.x == 0) {
      colmean[j] = mu;
      descale[j] = bound < 3.0e38f ? ldexpf(1.0f, -e) : __int_as_float(0x7fc00000);
    }
  }
  __syncthreads();
  const float mu = s_mu;
  const Scale sc(s_e);
  const int64_t k = (int64_t)blockIdx.x * kQChunk + 8 * threadIdx.x;
  int32_t q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (col >= 0 && k < np) {
    const float4* p = reinterpret_cast<const float4*>(Pf + (int64_t)col * np + k);
    const float4 a = p[0], b = p[1];
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    const double2* wv = reinterpret_cast<const double2*>(winv + (int64_t)slot * np + k);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const double2 w = wv[i];
      if (w.x != 0.0) q[2 * i] = __float2int_rn(sc(v[2 * i] - mu));
      if (w.y != 0.0) q[2 * i + 1] = __float2int_rn(sc(v[2 * i + 1] - mu));
    }
  }
  if (k < (int64_t)dt.stages * kStageK) store_digits(out, dt, j, k, q);
  // sums of integers, exact
  double t = (double)(((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7])));
  float none = 0.0f;
  __syncthreads();  // sh is read above
  block_sum_max(t, none, sh, shm);
  if (threadIdx.x == 0) qsum[j * nblk + blockIdx.x] = t;
}

// T[j, flips[k]] += dfill[k] * sum over the subset samples missing at that marker of v_c[j, i]: block
// (w, j) scans every sample's bit-map word w and accumulates the (at most 32) markers of that word in
// registers, then reduces them over the block in a fixed order.
__global__ void __launch_bounds__(kQThreads)
fp4_flip_t_kernel(const float* __restrict__ Pf, const float* __restrict__ colmean, int64_t np, int64_t nn,
                  const int32_t* __restrict__ cols, const ColState* __restrict__ st,
                  const SubsetSlot* __restrict__ slots, float* __restrict__ T, int64_t mg) {
  __shared__ float red[kQThreads / 32][32];
  const int64_t j = blockIdx.y;
  const int32_t col = cols[j];
  if (col < 0) return;
  const SubsetSlot sl = slots[st[col].pheno];
  const int w = blockIdx.x;
  if (w >= sl.W) return;
  float acc[32];
#pragma unroll
  for (int b = 0; b < 32; ++b) acc[b] = 0.0f;
  const uint32_t* bw = sl.bits + (int64_t)w * np;
  const float* p = Pf + (int64_t)col * np;
  const float mu = colmean[j];
  for (int64_t i = threadIdx.x; i < nn; i += kQThreads) {
    const uint32_t word = bw[i];
    if (word == 0u) continue;
    const float v = p[i] - mu;
#pragma unroll
    for (int b = 0; b < 32; ++b)
      if ((word >> b) & 1u) acc[b] += v;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int b = 0; b < 32; ++b) {
    float x = acc[b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == b) red[warp][b] = x;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const int b = threadIdx.x, k = 32 * w + b;
    if (k < sl.nflip) {
      float s = 0.0f;
      for (int q = 0; q < kQThreads / 32; ++q) s += red[q][b];
      T[j * mg + sl.flips[k]] += sl.dfill[k] * s;
    }
  }
}

// T' = d' .* (T - 2p' sum v_c) in place, and block maxima of |T'| (kQChunk markers each).  The sum of
// the quantised v_c is what the rounding of the mean leaves of it.
__global__ void __launch_bounds__(kQThreads)
fp4_tprime_kernel(float* __restrict__ T, int64_t mg, const int32_t* __restrict__ cols,
                  const ColState* __restrict__ st, const SubsetSlot* __restrict__ slots,
                  const double* __restrict__ qsum, int nsum, const float* __restrict__ descale1,
                  float* __restrict__ pmax, int nblk) {
  __shared__ double sh[kQThreads / 32];
  __shared__ float shm[kQThreads / 32];
  const int64_t j = blockIdx.y;
  const int32_t col = cols[j];
  const int64_t k = (int64_t)blockIdx.x * kQChunk + 8 * threadIdx.x;
  float mx = 0.0f;
  column_sum_max(qsum + j * nblk, nullptr, col >= 0 ? nsum : 0, sh, shm);
  const float sv = -(float)(sh[0] * (double)descale1[j]);
  if (col >= 0 && k < mg) {  // mg is a multiple of 128
    const float4* d = reinterpret_cast<const float4*>(slots[st[col].pheno].dprime + k);
    const float4* p = reinterpret_cast<const float4*>(slots[st[col].pheno].p2 + k);
    float4* t = reinterpret_cast<float4*>(T + j * mg + k);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4 x = t[h];
      const float4 y = d[h], z = p[h];
      x = make_float4(fmaf(z.x, sv, x.x) * y.x, fmaf(z.y, sv, x.y) * y.y, fmaf(z.z, sv, x.z) * y.z,
                      fmaf(z.w, sv, x.w) * y.w);
      t[h] = x;
      mx = fmaxf(mx, fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))));
    }
  }
  double none = 0.0;
  __syncthreads();  // sh is read above
  block_sum_max(none, mx, sh, shm);
  if (threadIdx.x == 0) pmax[j * nblk + blockIdx.x] = mx;
}

// T' as base-13 digits (padding columns zero), and the block partials of (2p')^T T' from the quantised
// values GEMM 2 multiplies, with 2p' in FP64: U - (2p')^T T' then sums to zero over the subset, as
// K_S v does, instead of carrying the rounding of 2p' and of the sum as a common shift.
__global__ void __launch_bounds__(kQThreads)
fp4_scale_digits_kernel(const float* __restrict__ T, int64_t mg, const int32_t* __restrict__ cols,
                        const ColState* __restrict__ st, const SubsetSlot* __restrict__ slots,
                        const float* __restrict__ pmax, int nblk, int nmax, DigitTile dt, uint8_t* __restrict__ out,
                        float* __restrict__ descale, double* __restrict__ part) {
  __shared__ double sh[kQThreads / 32];
  __shared__ float shm[kQThreads / 32];
  const int64_t j = blockIdx.y;
  const int32_t col = cols[j];
  const SubsetSlot* sl = col >= 0 ? &slots[st[col].pheno] : nullptr;
  column_sum_max(nullptr, pmax + j * nblk, col >= 0 ? nmax : 0, sh, shm);
  const int e = fixed_exponent(shm[0]);
  if (blockIdx.x == 0 && threadIdx.x == 0)
    descale[j] = shm[0] < 3.0e38f ? ldexpf(1.0f, -e) : __int_as_float(0x7fc00000);
  const Scale sc(e);
  const float inv = ldexpf(1.0f, -e);
  const int64_t k = (int64_t)blockIdx.x * kQChunk + 8 * threadIdx.x;
  double cf = 0.0;
  if (k < (int64_t)dt.stages * kStageK) {
    int32_t q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (sl && k < mg) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 t = *reinterpret_cast<const float4*>(T + j * mg + k + 4 * h);
        const double2* p = reinterpret_cast<const double2*>(sl->p2d + k + 4 * h);
        const double2 p01 = p[0], p23 = p[1];
        const float x[4] = {t.x, t.y, t.z, t.w};
        const double pp[4] = {p01.x, p01.y, p23.x, p23.y};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int32_t qi = __float2int_rn(sc(x[i]));
          q[4 * h + i] = qi;
          // |q| <= 2^24 is exact in FP32; a value that is not finite stays so in the sum
          cf = fma(pp[i], (double)(isfinite(x[i]) ? (float)qi * inv : x[i]), cf);
        }
      }
    }
    store_digits(out, dt, j, k, q);
  }
  float none = 0.0f;
  __syncthreads();  // shm is read above
  block_sum_max(cf, none, sh, shm);
  if (threadIdx.x == 0) part[j * nblk + blockIdx.x] = cf;
}

// K_S v on the subset: (U + dF T' - (2p')^T T') / M', written to column cols[j] of Y (zero outside the
// subset); padding columns are skipped.  The fill-flip term of sample i sums dfill[k] T'[j, flips[k]]
// over the flip markers it misses (set bits of the slot's word-major bit map), staged per column in
// shared memory, kFinF flips at a time, and added in ascending flip order.  (2p')^T T' is subtracted
// as two floats: its rounding to one would shift every sample alike.
constexpr int kFinF = 2048;

__global__ void __launch_bounds__(kQThreads)
fp4_finalize_kernel(const float* __restrict__ U, int64_t np, int64_t nn, const int32_t* __restrict__ cols,
                    const ColState* __restrict__ st, const SubsetSlot* __restrict__ slots,
                    const float* __restrict__ T, int64_t mg, const float* __restrict__ descale,
                    const double* __restrict__ part, int nblk, int nsum, const double* __restrict__ winv,
                    float* __restrict__ Yf) {
  __shared__ double sh[kQThreads / 32];
  __shared__ float shm[kQThreads / 32];
  __shared__ float tf[kFinF];
  const int64_t j = blockIdx.y;
  const int32_t col = cols[j];
  if (col < 0) return;
  const int slot = st[col].pheno;
  const SubsetSlot sl = slots[slot];
  column_sum_max(part + j * nblk, nullptr, nsum, sh, shm);
  const double c = sh[0];
  const int64_t k = (int64_t)blockIdx.x * kQChunk + 8 * threadIdx.x;
  unsigned live = 0u;
  float du[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (k < np) {
    const double2* wv = reinterpret_cast<const double2*>(winv + (int64_t)slot * np + k);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const double2 w = wv[i];
      if (w.x != 0.0) live |= 1u << (2 * i);
      if (w.y != 0.0) live |= 2u << (2 * i);
    }
  }
  const float inv = descale[j];  // a power of two, or NaN
  const Scale sc(inv > 0.0f ? -ilogbf(inv) : 0);
  for (int f0 = 0; f0 < sl.nflip; f0 += kFinF) {
    const int fn = sl.nflip - f0 < kFinF ? sl.nflip - f0 : kFinF;
    __syncthreads();
    for (int q = threadIdx.x; q < fn; q += kQThreads)  // T' as GEMM 2 multiplied it
      tf[q] = sl.dfill[f0 + q] * (rintf(sc(T[j * mg + sl.flips[f0 + q]])) * inv);
    __syncthreads();
    const int w0 = f0 / 32, wn = (fn + 31) / 32;
    for (int i = 0; i < 8; ++i) {
      if (!((live >> i) & 1u)) continue;
      const uint32_t* bw = sl.bits + (int64_t)w0 * np + k + i;
      float d = du[i];
      for (int w = 0; w < wn; ++w) {
        uint32_t word = bw[(int64_t)w * np];
        while (word) {
          const int b = __ffs(word) - 1;
          word &= word - 1u;
          d += tf[32 * w + b];
        }
      }
      du[i] = d;
    }
  }
  if (k >= np) return;
  const float ch = (float)c, cl = (float)(c - (double)ch), inv_mf = (float)sl.inv_m;
  float4* o = reinterpret_cast<float4*>(Yf + (int64_t)col * np + k);
  const float4* u = reinterpret_cast<const float4*>(U + j * np + k);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float4 x = u[h];
    const float in[4] = {x.x, x.y, x.z, x.w};
    float y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      y[i] = (live >> (4 * h + i)) & 1u ? ((in[i] - ch) - cl + du[4 * h + i]) * inv_mf : 0.0f;
    o[h] = make_float4(y[0], y[1], y[2], y[3]);
  }
}

// ----------------------------------------------------------------------------------- products
// Columns per tile for a launch over ncols columns.
int fp4_tile_cols(int64_t ncols) {
  if (ncols <= 16) return 16;
  if (ncols <= 32) return 32;
  if (ncols <= 48) return 48;
  return 64;
}

static cudaError_t fp4_gemm(const void* G, int64_t rows, int64_t k, const void* Bq, int64_t ncols, int ct, float* D,
                            int64_t ldd, const float* descale, cudaStream_t s) {
  if (rows <= 0 || k <= 0 || ncols <= 0 || ncols % ct != 0 || !G || !Bq) return cudaErrorInvalidValue;
  const int stages = fp4_stages(k);
  CUtensorMap a, b;
  if (!fp4_map(&a, G, fp4_matrix_bytes(rows, k), kAStage / kMapRow) ||
      !fp4_map(&b, Bq, ncols * (int64_t)stages * 672, (uint32_t)(336 * ct / kMapRow)))
    return cudaErrorInvalidValue;
  int* err = tc_error_flag();
  if (!err) return cudaErrorInvalidValue;
  const int nt = (int)(ncols / ct);
  const int64_t tiles = (rows + 255) / 256 * nt;
  switch (ct) {
    case 16: return launch_fp4<16, 6, kProduct>(a, b, stages, rows, tiles, nt, D, ldd, descale, {}, err, s);
    case 32: return launch_fp4<32, 4, kProduct>(a, b, stages, rows, tiles, nt, D, ldd, descale, {}, err, s);
    case 48: return launch_fp4<48, 7, kProduct>(a, b, stages, rows, tiles, nt, D, ldd, descale, {}, err, s);
    case 64: return launch_fp4<64, 6, kProduct>(a, b, stages, rows, tiles, nt, D, ldd, descale, {}, err, s);
    default: return cudaErrorInvalidValue;
  }
}

static int chunks(int64_t n) { return (int)((n + kQChunk - 1) / kQChunk); }
// one more than the vectors' chunks: a digit operand's K is padded to whole stages
int fp4_nblk(int64_t np, int64_t mg) { return chunks(np > mg ? np : mg) + 1; }

cudaError_t fp4_product(const void* Gmm, const void* Gsm, const float* Pf, int64_t np, int64_t nn, int64_t mg,
                        int64_t m, const int32_t* cols, int64_t ncols, int ct, const ColState* st,
                        const SubsetSlot* slots, const double* winv, int max_w, const Fp4Scratch& w, float* Yf,
                        cudaStream_t s, int* launches) {
  const int nblk = fp4_nblk(np, mg);
  const DigitTile dv{ct, fp4_stages(nn)}, dt{ct, fp4_stages(m)};
  const int nsum = chunks(np), nmax = chunks(mg);
  const int nv = chunks((int64_t)dv.stages * kStageK), nt = chunks((int64_t)dt.stages * kStageK);
  const unsigned y = (unsigned)ncols;
  fp4_sums_kernel<<<dim3((unsigned)nsum, y), kQThreads, 0, s>>>(Pf, np, cols, w.part, w.pmax, nblk);
  fp4_center_digits_kernel<<<dim3((unsigned)nv, y), kQThreads, 0, s>>>(Pf, np, cols, st, slots, winv, w.part, w.pmax,
                                                                       nblk, nsum, dv, static_cast<uint8_t*>(w.Vq),
                                                                       w.mean, w.descale1, w.qsum);
  cudaError_t e = fp4_gemm(Gmm, mg, nn, w.Vq, ncols, ct, w.T, mg, w.descale1, s);
  if (e != cudaSuccess) return e;
  if (max_w > 0)
    fp4_flip_t_kernel<<<dim3((unsigned)max_w, y), kQThreads, 0, s>>>(Pf, w.mean, np, nn, cols, st, slots, w.T, mg);
  fp4_tprime_kernel<<<dim3((unsigned)nmax, y), kQThreads, 0, s>>>(w.T, mg, cols, st, slots, w.qsum, nv, w.descale1,
                                                                w.pmax, nblk);
  fp4_scale_digits_kernel<<<dim3((unsigned)nt, y), kQThreads, 0, s>>>(w.T, mg, cols, st, slots, w.pmax, nblk, nmax, dt,
                                                                      static_cast<uint8_t*>(w.Tq), w.descale2, w.part);
  e = fp4_gemm(Gsm, np, m, w.Tq, ncols, ct, w.U, np, w.descale2, s);
  if (e != cudaSuccess) return e;
  fp4_finalize_kernel<<<dim3((unsigned)nsum, y), kQThreads, 0, s>>>(w.U, np, nn, cols, st, slots, w.T, mg, w.descale2,
                                                                    w.part, nblk, nt, winv, Yf);
  *launches = max_w > 0 ? 8 : 7;
  return cudaGetLastError();
}

// ----------------------------------------------------------------------------------- the GRM
// K = Z Z' / M from the packed GRM genotypes, z = (g - 2p) / sd:
//
//   M K_ij = sum_m D_m g_im g_jm - a_i - a_j + c0,  D = 1/sd^2,  a_i = sum_m 2p_m D_m g_im,  c0 = sum_m 4p_m^2 D_m
//
// with D_m fixed to integers (2 D_m <= 2^24).  The rows of B are samples: element m of row j is D_m g_jm, one of
// 0, D_m, 2 D_m, in base-13 digits; the sums are exact, and so is the subtraction of a_i and a_j, which cancels
// most of them: only D's rounding (2^-25 of its largest value) and the entry's two to FP32 (its sum, and the sum's
// product with the scale) remain.
// Against split-BF16's four products (off-diagonal error 4e-8 of entries of RMS 2.6e-3 at 100k x 150k, and row
// sums off by n times its bias) this takes seven FP4 products, 1.2 BF16 ones' tensor time.
namespace {

constexpr int kSyrkTile = 64;

// Digits of D_m g_jm for a column tile of 64 samples and one stage of 192 markers: thread = (sample, chunk of 32
// markers), its masks (one copy, two copies) applied to the stage's digit words.
// words: [stage][digit][24 groups of 8 markers] of (codes of D, codes of 2 D)
__global__ void __launch_bounds__(384)
fp4_syrk_digits_kernel(const uint8_t* __restrict__ packed, int64_t pitch, int64_t m, int64_t n, int stages,
                       const uint2* __restrict__ words, uint8_t* __restrict__ out) {
  __shared__ uint8_t sc[kStageK][17];
  __shared__ uint2 sw[kDigits * 24];
  const int ks = blockIdx.x;
  const int64_t tile = blockIdx.y;
  for (int t = threadIdx.x; t < kStageK * 16; t += blockDim.x) {
    const int mm = t >> 4, b = t & 15;
    const int64_t mk = (int64_t)ks * kStageK + mm, off = tile * 16 + b;
    sc[mm][b] = mk < m && off < pitch ? packed[mk * pitch + off] : 0xFF;
  }
  for (int t = threadIdx.x; t < kDigits * 24; t += blockDim.x) sw[t] = words[(int64_t)ks * (kDigits * 24) + t];
  __syncthreads();
  const int j = threadIdx.x & 63, chunk = threadIdx.x >> 6;
  const bool live = tile * 64 + j < n;
  uint32_t m1[4], m2[4];
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    uint32_t a = 0, b = 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const uint32_t f = (sc[chunk * 32 + 8 * w + e][j >> 2] >> (2 * (j & 3))) & 3u;
      a |= (f == 2u ? 15u : 0u) << (4 * e);
      b |= (f == 0u ? 15u : 0u) << (4 * e);
    }
    m1[w] = live ? a : 0u;
    m2[w] = live ? b : 0u;
  }
  const DigitTile dt{kSyrkTile, stages};
  const DigitColumn dc = digit_column(dt, j);
  uint8_t* o = out + tile * (int64_t)stages * (672 * kSyrkTile) + (int64_t)ks * (672 * kSyrkTile) + chunk * 128;
#pragma unroll
  for (int d = 0; d < kDigits; ++d) {
    uint32_t x[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint2 c = sw[d * 24 + chunk * 4 + w];
      x[w] = (c.x & m1[w]) | (c.y & m2[w]);
    }
    const int r = dc.r + d, rank = r >= dc.hn ? 1 : 0, row = 112 * dc.h + r - rank * dc.hn;
    *reinterpret_cast<uint4*>(o + rank * (336 * kSyrkTile) + (row >> 3) * kGroupStage + (row & 7) * 16) =
        make_uint4(x[0], x[1], x[2], x[3]);
  }
}

// The two columns of 2p_m D_m 2^16 = hi 2^18 + lo as digits of a 16-column tile (the others zero).
__global__ void fp4_shift_digits_kernel(const int2* __restrict__ hilo, int64_t m, int stages, uint8_t* __restrict__ out) {
  const int64_t k = 8 * ((int64_t)blockIdx.x * blockDim.x + threadIdx.x);
  if (k >= (int64_t)stages * kStageK) return;
  const DigitTile dt{16, stages};
  for (int j = 0; j < 16; ++j) {
    int32_t q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      q[i] = 0;
      if (j < 2 && k + i < m) q[i] = j == 0 ? hilo[k + i].x : hilo[k + i].y;
    }
    store_digits(out, dt, j, k, q);
  }
}

// a_i = (hi_i 2^18 + lo_i) / 2^16, rounded (the shifted sum stays below 2^62)
__global__ void fp4_shift_kernel(const long long* __restrict__ sums, int64_t ld, int64_t n, long long* __restrict__ shift) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  shift[i] = ((sums[i] << 18) + sums[ld + i] + (1ll << 15)) >> 16;
}

}  // namespace

// Bound on max D times the RMS of 1/D, to which the entries' RMS error is in proportion (where the line lies: sg_grm_build).
double fp4_syrk_spread(int64_t m, bool split_bf16) {
  if (split_bf16) return 80.0;
  return std::max(0.6 * std::sqrt((double)m), m >= 128 ? 24.0 : 0.0);
}

// Bytes of a build's scratch (see fp4_syrk), and whether D's range lets integers of 24 bits hold it: the markers of the
// smallest D then keep an error of 2^-25 ``range`` relative at most.
Fp4SyrkPlan fp4_syrk_plan(const double* weight, int64_t m, int64_t np, double range) {
  Fp4SyrkPlan p;
  double lo = 1e300, hi = 0.0;
  for (int64_t i = 0; i < m; ++i) {
    const double d = weight[i];
    if (d > 0.0) {
      lo = d < lo ? d : lo;
      hi = d > hi ? d : hi;
    }
  }
  if (m <= 0 || !(hi > 0.0) || !(hi < 1e30) || hi > range * lo || fp4_stages(m) > kSegStages) return p;
  int e = 0;
  frexp(hi, &e);  // hi < 2^e
  p.exponent = 23 - e;
  p.ok = true;
  const int64_t stages = fp4_stages(m);
  auto add = [&](int64_t bytes) {
    const int64_t at = p.bytes;
    p.bytes += round_up(bytes, 256);
    return at;
  };
  p.off_a = add(fp4_matrix_bytes(np, m));
  p.off_b = add(round_up(np, kSyrkTile) * stages * 672);
  p.off_shift_b = add(16 * stages * 672);
  p.off_sums = add(16 * np * 8);
  p.off_shift = add(np * 8);
  p.off_words = add(stages * kDigits * 24 * 8);
  p.off_hilo = add(m * 8);
  // lower-triangle tiles: groups of 8 row tiles (256 rows) sweep the column tiles together, so the pairs
  // resident at one time share a few panels of either operand in L2
  const int64_t nrt = (np + 255) / 256;
  for (int64_t g0 = 0; g0 < nrt; g0 += 8) {
    const int64_t g1 = g0 + 8 < nrt ? g0 + 8 : nrt;
    for (int64_t bt = 0; bt * kSyrkTile < np && bt * kSyrkTile < g1 * 256; ++bt)
      for (int64_t rt = g0; rt < g1; ++rt)
        if (bt * kSyrkTile < rt * 256 + 256) {
          p.tiles.push_back((int32_t)rt);
          p.tiles.push_back((int32_t)bt);
        }
  }
  p.off_tiles = add((int64_t)p.tiles.size() * 4);
  return p;
}

// K = (1/m) sum_m weight_m (g_i - centre_m) (g_j - centre_m) (np x np, FP32, both triangles) from packed
// genotypes (m x pitch bytes), in the plan's scratch.  Returns after the work has run.
cudaError_t fp4_syrk(const Fp4SyrkPlan& p, void* scratch, const uint8_t* packed, int64_t pitch, const double* weight,
                     const double* centre, int64_t m, int64_t n, int64_t np, float* K, cudaStream_t s) {
  uint8_t* base = static_cast<uint8_t*>(scratch);
  const int stages = fp4_stages(m);
  // host tables: D_m's digit words, (hi, lo) of 2p_m D_m 2^16, c0
  std::vector<uint32_t> words((size_t)stages * kDigits * 24 * 2, 0u);
  std::vector<int32_t> hilo((size_t)m * 2);
  double c0 = 0.0;
  for (int64_t i = 0; i < m; ++i) {
    const double two_p = centre[i];
    const int32_t D = (int32_t)std::llrint(std::ldexp(weight[i], p.exponent));
    const uint32_t c1 = digit_codes(D), c2 = digit_codes(2 * D);
    const int64_t ks = i / kStageK, g = (i % kStageK) / 8, e = i % 8;
    for (int t = 0; t < kDigits; ++t) {
      uint32_t* w = &words[((size_t)(ks * kDigits + t) * 24 + g) * 2];
      w[0] |= ((c1 >> (4 * t)) & 15u) << (4 * e);
      w[1] |= ((c2 >> (4 * t)) & 15u) << (4 * e);
    }
    const long long h = std::llrint(std::ldexp((double)D * two_p, 16));
    hilo[2 * i] = (int32_t)(h >> 18);
    hilo[2 * i + 1] = (int32_t)(h & ((1 << 18) - 1));
    c0 += (double)D * two_p * two_p;
  }
  cudaError_t e = cudaMemcpyAsync(base + p.off_words, words.data(), words.size() * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(base + p.off_hilo, hilo.data(), hilo.size() * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(base + p.off_tiles, p.tiles.data(), p.tiles.size() * 4, cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess) return e;
  const int64_t rs = (np + 255) / 256 * 2;
  launch_fp4_gbuild_sm(packed, pitch, nullptr, m, n, stages, rs, base + p.off_a, s);
  const int64_t nbt = (np + kSyrkTile - 1) / kSyrkTile;
  fp4_syrk_digits_kernel<<<dim3((unsigned)stages, (unsigned)nbt), 384, 0, s>>>(
      packed, pitch, m, n, stages, reinterpret_cast<const uint2*>(base + p.off_words), base + p.off_b);
  fp4_shift_digits_kernel<<<(unsigned)((stages * (kStageK / 8) + 127) / 128), 128, 0, s>>>(
      reinterpret_cast<const int2*>(base + p.off_hilo), m, stages, base + p.off_shift_b);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  CUtensorMap a, b, bs;
  int* err = tc_error_flag();
  if (!err || !fp4_map(&a, base + p.off_a, fp4_matrix_bytes(np, m), kAStage / kMapRow) ||
      !fp4_map(&b, base + p.off_b, round_up(np, kSyrkTile) * (int64_t)stages * 672, 336 * kSyrkTile / kMapRow) ||
      !fp4_map(&bs, base + p.off_shift_b, 16 * (int64_t)stages * 672, 336 * 16 / kMapRow))
    return cudaErrorInvalidValue;
  long long* sums = reinterpret_cast<long long*>(base + p.off_sums);
  long long* shift = reinterpret_cast<long long*>(base + p.off_shift);
  e = launch_fp4<16, 6, kSums>(a, bs, stages, np, (np + 255) / 256, 1, sums, np, nullptr, {}, err, s);
  if (e != cudaSuccess) return e;
  fp4_shift_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(sums, np, n, shift);
  const SyrkArgs sy{reinterpret_cast<const int2*>(base + p.off_tiles), shift, std::llrint(c0),
                    (float)(std::ldexp(1.0, -p.exponent) / (double)m), n};
  e = launch_fp4<kSyrkTile, 6, kSyrk>(a, b, stages, np, (int64_t)p.tiles.size() / 2, 1, K, np, nullptr, sy, err, s);
  if (e != cudaSuccess) return e;
  return tc_check_error(s);
}

}  // namespace sg
