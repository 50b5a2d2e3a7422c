// gemm_oz.cu -- the FP64 matrix update on the tensor cores:
//     C (m x n) -= A (m x k) * B (k x n)
// for complex128 or real double, column-major, to FP64 accuracy entry by entry,
// with tcgen05.mma (kind::f16) on integer slices of the operands (the error-free
// splitting of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication and
// its applications", Numer. Algorithms 59, 2012).
//
// Each row of A and each column of B is scaled by the power of two above its
// largest entry and rounded to a 71-bit fixed-point number, written as nine
// balanced base-256 digits (-128 .. 128, exact in bf16).  The product of two
// digit matrices is an integer; its FP32 accumulator is exact while it stays
// within 2^24, that is over 1024 products of at most 2^14.  The pairs (i, j)
// of slices with i + j = d share the weight 2^-(8d - 2), so they add up in one
// accumulator, as many pairs as the 1024 products allow; the groups d = 2 .. 9
// (36 pairs) are drained into one 64-bit integer per output, which is rounded to
// FP64 once (integer arithmetic) and subtracted from C.
//
// What fixed point leaves out is a fraction of (row maximum) x (column maximum),
// where FP64 products lose a fraction of each |a_ik b_kj|.  The two differ where
// a row's large entries meet a column's small ones: rows of different scale, a
// weakly coupled set of unknowns, low frequencies (of a dielectric, electric and
// magnetic currents in turn).  So one more slice holds the entries' sizes as
// ordinary bf16 numbers, and its product, the first of a tile, is every output's
// own sum S = sum |a_ik| |b_kj| in units of the two maxima.  Outputs with
//   S >= 1      are summed in units of 2^-53, with
//   S <  1      in units of 2^-62 (modulo 2^64: the sum is below 2^62 of them);
//   S <  2^-8   add the pairs of d = 10 to their tile, last;
//   S <  2^-10  are left to FP64 multiplications by the draining warp where it has
//               few (FEW); where it has more, its outputs with
//     S < 2^-8  are summed in units of 2^-70, with
//     S < 2^-16 in units of 2^-78 (and d = 11 is added),
//     S < 2^-20 left to FP64 multiplications.
// Whatever is left out is then a rounding or two of sum |a_ik| |b_kj|, which FP64
// chains of 128 to 512 products exceed.  Measured, N = 400, largest |P A - L U| /
// |L||U| of an LU, in units of 2^-53:
//                                          seven digits alone   now   LAPACK
//   normal entries                                  1.8         1.8     1.9
//   rows scaled over 1e12, the smallest first       300         1.8     1.7
//   over 1e18, 1e30                             2.3e4, 7.7e7  2.1, 1.4  1.8, 2.1
//   two sets coupled by 1e-6, 1e-12             5.9e4, 8.2e10 2.8, 2.5  3.3, 2.8
// and of an update by itself, entries over 2^60, k = 7 .. 256: 1 to 4, chains of
// FP64 FMAs 2 to 15.  Error for normal entries, k = 256: 4.4e-18 of |a| |b| root
// mean square, FP64 FMAs 4.3e-17; backward error of an LU of normal entries,
// N = 768: 3.6e-15 (LAPACK 6.3e-15, FP64 updates 5.6e-15).
//
// Time, k = 256 complex: m = n = 3584 0.97 ms, 27 TFLOP/s FP64 (0.87 with seven
// digits alone), against 0.74 TFLOP/s for the SIMT FP64 update; 1653 306 us (267);
// 480 x 64, k = 64 33 us (31); real 3584 401 us (402).  LU of dielectric spheres,
// N = 3840, kR = 2, 0.5, 0.1: 37, 41, 57 ms; 36 with seven digits alone, 290 with SIMT
// updates; with every output below 2^-10 left to FP64 37, 59 and, at 0.05 (76 now),
// 182.
//
// What bounds it: large updates, the draining warps' instructions -- ncu, m = n =
// 3584, k = 256: tensor pipe 43 % active, of the drain's stalls a quarter waits for
// instructions (64 outputs of a thread are 64 copies of the code) and a third for
// TMEM, C and spilled words; one conversion for every exponent in place of three
// branches 1.04 -> 0.97 ms.  Small ones, the single-thread TMA and MMA issuers'
// instructions per k-step.  Output tiles are walked in bands of 16 rows of tiles: with
// columns of 118 the slices of A no longer fit the L2 (m = n = 15104, k = 128: 12.8 ->
// 10.7 ms).  The FP64 pipe it replaces runs 2 FMAs per cycle and SM; outputs left to it
// take as long as gemm_simt took.
//
// A row or column that holds an infinity or NaN makes its row or column of C
// NaN (the digits are zero there).
#include <cuda_bf16.h>
#include <algorithm>
#include <cstdlib>
#include "bem_math.cuh"
#include "gbem_internal.h"
#include "tc_ptx.cuh"

namespace gbem {

namespace oz {
constexpr int NS = 9;             // slices (base-256 digits); slice NS + 1 holds the sizes
constexpr int STEPS = 11;         // groups of slice pairs: sizes, d = 9 .. 2, and d = 10, 11 where they are called for
// outputs by the sum of their products' sizes (see above)
constexpr float S_FINE = 1.0f, S_10 = 0x1p-8f, S_FEW = 0x1p-10f, S_11 = 0x1p-16f, S_FP64 = 0x1p-20f;
constexpr int FEW = 8;            // outputs below S_FEW that a warp leaves to FP64 rather than go below units of 2^-62
constexpr int KMAX = 512;         // real products per output and slice pair
constexpr int ACC_TERMS = 1024;   // products that add up exactly: 1024 * 2^14 = 2^24
constexpr int BM = 128, BK = 64;
// k-blocks of BK per stage, one TMA instruction per operand: what bounds a
// k-step is the instructions of the producer and the MMA issuer (about 0.25 us
// for a wait, two TMA copies and a commit), not the ring's depth or the MMAs
// (m = n = 1653, k = 256: 232 us with 2 blocks, 273 with 1, 315 with 4, whose
// ring is one stage deep)
constexpr int KB = 2;
// output tile BM x BN: its TMA ring and instruction descriptor
template <int BN> struct Tile {
  static constexpr int STAGES = BN == 128 ? 3 : 5;
  // a stage holds KB k-blocks of A, then of B
  static constexpr int A_BLK = BM * BK * 2, B_BLK = BN * BK * 2;
  static constexpr int A_BYTES = KB * A_BLK, B_BYTES = KB * B_BLK, STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
  static constexpr uint32_t IDESC = idesc_bf16(BM, BN);
  static_assert((2 * STAGES + 6) * 8 + 4 <= 256, "barrier area");
  static_assert(B_BLK % 1024 == 0, "swizzle atoms");
};
constexpr int EXP_BAD = 1 << 20;  // scale exponent of a row or column that is not finite
constexpr int BAND = 16;          // rows of output tiles walked together (8 and 32 within 1 %)
constexpr int VECS = 16;          // rows of A (columns of B) per packing CTA
}  // namespace oz

// exponent field (at least 1) of a double's high word
__device__ __forceinline__ int exp_field(unsigned hi) { return max((int)((hi >> 20) & 0x7ffu), 1); }

// |x| < 2^(F - 1022) as a 71-bit fixed-point number, round(|x| 2^(71 - (F - 1022))):
// its leading 39 and its last 32 bits, in balanced digits -- bytes 0..3 of hi are the
// digits 5..2 plus 128, above them the top digit; bytes 0..3 of lo the digits 9..6
// plus 128 -- and its size as a bf16 number in units of 2^(F - 1022): no entry but
// zero has size zero, so that a sum of sizes is zero only where every product is
struct OzDigits { unsigned long long hi; unsigned lo; unsigned short size; };
__device__ __forceinline__ OzDigits oz_digits(double x, int F) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int raw = (int)((b >> 52) & 0x7ffu), d = F - max(raw, 1);  // d >= 0
  unsigned long long M = b & 0xfffffffffffffull;
  if (raw) M |= 1ull << 52;
  unsigned long long hi, lo;
  if (d <= 18) {
    hi = M >> (14 + d);
    lo = M << (18 - d) & 0xffffffffull;
  } else {
    lo = d < 74 ? (M + (1ull << (d - 19))) >> (d - 18) : 0;
    hi = lo >> 32;
    lo &= 0xffffffffull;
  }
  lo += 0x80808080ull;
  OzDigits r;
  r.lo = (unsigned)lo;
  r.hi = hi + (lo >> 32) + 0x80808080ull;
  const float v = (float)M * __int_as_float((74 - min(d, 60)) << 23);  // M 2^-53 2^-d
  r.size = M ? __bfloat16_as_ushort(__float2bfloat16_rn(fmaxf(v, 0x1p-60f))) : (unsigned short)0;
  return r;
}

// step of a tile (0: the sizes; 1 .. 8: d = 9 .. 2; 9, 10: d = 10, 11) -> its slice pairs (i, j), i0 <= i < i1, j = sum - i
struct OzGroup { int i0, i1, sum; };
// (d = 10 without the ninth digits where units of 2^-62 are the finest: narrow)
__device__ __forceinline__ OzGroup oz_group(int step, bool narrow) {
  if (step == 0) return {oz::NS + 1, oz::NS + 2, 2 * oz::NS + 2};
  const int d = step < 9 ? 10 - step : step + 1;
  const int cut = d == 10 && narrow ? 1 : 0;
  return {max(1, d - oz::NS) + cut, min(oz::NS + 1, d) - cut, d};
}

// The digits of A's rows (part 0) and B's columns (part 1), one launch: CTAs
// [0, na) take 16 rows of A each, the others 16 columns of B.  The vectors
// are staged in shared memory (coalesced), their largest exponent is found,
// and each vector's digits and sizes are written slice by slice,
// out[s][row][Kp], zero beyond kreal.  A complex row of A is [Re | Im]; a complex column j of
// B makes rows 2j = [Re | -Im] and 2j + 1 = [Im | Re], whose products with it
// are the real and imaginary part.
template <bool CPLX>
__global__ void __launch_bounds__(256) oz_pack(const double* A, long long lda, int m, const double* B, long long ldb,
                                               int n, int k, int Kp, int na, __nv_bfloat16* outA, __nv_bfloat16* outB,
                                               int* ea, int* eb) {
  pdl_wait();
  pdl_trigger();
  constexpr int W = CPLX ? 2 : 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* t = reinterpret_cast<double*>(smem_raw);  // [k][17][W]
  __shared__ unsigned red[oz::VECS][17];
  __shared__ int vexp[oz::VECS];
  const bool isB = (int)blockIdx.x >= na;
  const int v0 = ((int)blockIdx.x - (isB ? na : 0)) * oz::VECS;
  const int nv = min(oz::VECS, (isB ? n : m) - v0);
  const int tid = threadIdx.x;
  for (int q = tid; q < oz::VECS * k; q += 256) {
    const int v = isB ? q / k : q % oz::VECS, kk = isB ? q % k : q / oz::VECS;
    double x = 0.0, y = 0.0;
    if (v < nv) {
      const long long o = isB ? kk + (long long)(v0 + v) * ldb : (v0 + v) + (long long)kk * lda;
      if (CPLX) {
        const double2 z = reinterpret_cast<const double2*>(isB ? B : A)[o];
        x = z.x; y = z.y;
      } else {
        x = (isB ? B : A)[o];
      }
    }
    t[(kk * 17 + v) * W] = x;
    if (CPLX) t[(kk * 17 + v) * W + 1] = y;
  }
  __syncthreads();
  {
    const int v = tid & 15, part = tid >> 4;
    unsigned mx = 0;
    for (int kk = part; kk < k; kk += 16)
      for (int c = 0; c < W; c++)
        mx = max(mx, (unsigned)__double2hiint(t[(kk * 17 + v) * W + c]) & 0x7fffffffu);
    red[v][part] = mx;
  }
  __syncthreads();
  if (tid < oz::VECS) {
    unsigned mx = 0;
    for (int p = 0; p < 16; p++) mx = max(mx, red[tid][p]);
    const bool bad = mx >= 0x7ff00000u;
    const int F = exp_field(mx);
    vexp[tid] = bad ? -1 : F;
    if (tid < nv) (isB ? eb : ea)[v0 + tid] = bad ? oz::EXP_BAD : F - 1022;
  }
  __syncthreads();
  const int groups = Kp >> 2;  // 4 digits per 8-byte store
  const int rpv = (isB && CPLX) ? 2 : 1;
  const int nrows = nv * rpv;
  const long long rows = (long long)(isB ? n : m) * rpv;
  __nv_bfloat16* out = isB ? outB : outA;
  for (int q = tid; q < nrows * groups; q += 256) {
    const int r = q / groups, g = q - r * groups;
    const int v = rpv == 2 ? r >> 1 : r, odd = rpv == 2 ? r & 1 : 0;
    const int F = vexp[v];
    OzDigits z[4];
    unsigned neg = 0;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const int p = 4 * g + e;
      double x = 0.0;
      if (CPLX) {
        const int seg = p >= k, kk = p - (seg ? k : 0);
        if (kk < k) {
          if (!isB) x = t[(kk * 17 + v) * 2 + seg];
          else {
            x = t[(kk * 17 + v) * 2 + (seg ^ odd)];
            if (seg && !odd) neg |= 1u << e;
          }
        }
      } else if (p < k) {
        x = t[p * 17 + v];
      }
      if (F < 0) x = 0.0;
      neg ^= (unsigned)(__double2hiint(x) < 0) << e;
      z[e] = oz_digits(x, F < 0 ? 1 : F);
    }
#pragma unroll
    for (int s = 0; s <= oz::NS; s++) {  // slice s holds digit s + 1 (the top one first), the last the sizes
      unsigned short w[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int dg = s == 0 ? (int)(z[e].hi >> 32)
                              : (int)((s < 5 ? z[e].hi >> (8 * (4 - s)) : (unsigned long long)(z[e].lo >> (8 * (8 - min(s, 8))))) & 255) - 128;
        w[e] = s == oz::NS ? z[e].size : (unsigned short)(__float_as_uint((float)((neg >> e) & 1u ? -dg : dg)) >> 16);
      }
      uint2 pk;
      pk.x = (unsigned)w[0] | ((unsigned)w[1] << 16);
      pk.y = (unsigned)w[2] | ((unsigned)w[3] << 16);
      *reinterpret_cast<uint2*>(out + ((long long)s * rows + (long long)v0 * rpv + r) * Kp + 4 * g) = pk;
    }
  }
}

// T 2^e rounded to 53 bits (fewer below 2^-1022; above the range infinite; NaN for
// the exponent of a row or column that is not finite), in integer arithmetic: the
// FP64 pipe (2 operations per cycle and SM) is left with the one subtraction.  One
// path for every exponent: a drain warp runs its 64 copies once a tile, and what it
// waits for most is instructions.
__device__ __forceinline__ double int_to_double(long long T, int e) {
  const unsigned long long a = T < 0 ? 0ull - (unsigned long long)T : (unsigned long long)T;
  const int lz = __clzll((long long)a);
  const unsigned long long m = a << (lz & 63);
  const int E = 1023 + 63 - 1 + e - lz;  // the exponent field, less what q brings
  const int r = 11 - max(min(E, 0), -53);
  const unsigned long long q = ((m >> (r - 1)) + 1) >> 1;  // 2^52 .. 2^53, less where E < 0
  unsigned long long b = ((unsigned long long)max(E, 0) << 52) + q;
  if (E > 2045) b = 0x7ff0000000000000ull;
  if (!a || E < -53) b = 0;
  b |= (unsigned long long)T & 0x8000000000000000ull;
  if (e > oz::EXP_BAD / 2) b = 0x7ff8000000000000ull;
  return __longlong_as_double((long long)b);
}

// the t-th output tile of mt x (ntiles / mt)
struct OzTile { int m, n; };
__device__ __forceinline__ OzTile oz_tile(int t, int mt, int ntiles) {
  const int nt = ntiles / mt, b = t / (oz::BAND * nt), r = t - b * oz::BAND * nt, h = min(oz::BAND, mt - b * oz::BAND);
  return {b * oz::BAND + r % h, r / h};
}

// x 2^s modulo 2^64, 0 <= s <= 64
__device__ __forceinline__ unsigned long long shl64(long long x, int s) {
  unsigned long long y;
  asm("shl.b64 %0, %1, %2;" : "=l"(y) : "l"(x), "r"(s));
  return y;
}

// C(row, j) -= sum_k A(row, k) B(k, j) in FP64 for a warp's outputs marked in need
// (bit c: its real column c; lane: its row).  Many of a column: each lane its own
// row; few: the lanes share the products of one after the other.
template <bool CPLX>
__device__ __noinline__ void oz_fp64(double* C, long long ldc, const double* A, long long lda, const double* B, long long ldb,
                                     int m, int n, int k, int row, int j0, unsigned need) {
  constexpr int W = CPLX ? 2 : 1;
  const int lane = threadIdx.x & 31, row0 = row - lane;
  auto term = [&](int r, int j, int kk, double& x, double& y) {
    const double* a = A + W * ((long long)r + (long long)kk * lda);
    const double* b = B + W * ((long long)kk + (long long)j * ldb);
    if (CPLX) {
      const double2 u = *reinterpret_cast<const double2*>(a), v = *reinterpret_cast<const double2*>(b);
      x = fma(-u.y, v.y, fma(u.x, v.x, x));
      y = fma(u.y, v.x, fma(u.x, v.y, y));
    } else {
      x = fma(*a, *b, x);
    }
  };
  auto put = [&](int r, int j, double x, double y) {
    double* p = C + W * ((long long)r + (long long)j * ldc);
    p[0] -= x;
    if (CPLX) p[W - 1] -= y;
  };
  for (int c = 0; c < 32; c += W) {
    const int j = j0 + c / W;
    if (j >= n) break;
    const bool mine = (need >> c) & (W == 2 ? 3u : 1u);
    unsigned rows = __ballot_sync(0xffffffffu, mine);
    if (__popc(rows) > 8) {
      if (mine) {
        double x = 0.0, y = 0.0;
#pragma unroll 4
        for (int kk = 0; kk < k; kk++) term(row, j, kk, x, y);
        put(row, j, x, y);
      }
      __syncwarp();
    } else {
      for (; rows; rows &= rows - 1) {
        const int r = row0 + __ffs(rows) - 1;
        double x = 0.0, y = 0.0;
        for (int kk = lane; kk < k; kk += 32) term(r, j, kk, x, y);
        for (int o = 16; o > 0; o >>= 1) {
          x += __shfl_xor_sync(0xffffffffu, x, o);
          if (CPLX) y += __shfl_xor_sync(0xffffffffu, y, o);
        }
        if (lane == 0) put(r, j, x, y);
      }
    }
  }
}

// One CTA per SM walks the 128 x BN output tiles (columns counted as reals;
// in bands of BAND rows of tiles, m fastest, so the CTAs of a wave share their B
// tiles and a band of A).  Warp 0: TMA producer;
// warp 1: TMEM and MMA issue; warps 2-9: drain.  A tile's accumulators follow
// one another through two BN-column TMEM buffers: the MMAs of the next run
// while the drain warps add the last one into their 64-bit integers (one row
// and BN / 2 columns per thread).  The sizes come first: by the end of a tile its
// draining warps have long decided whether d = 10 and 11 follow.  pairs: slice pairs
// per accumulator.  A, B: the operands themselves, for the outputs left to FP64.
template <bool CPLX, int BN>
__global__ void __launch_bounds__(320, 1) oz_gemm_kernel(const __grid_constant__ CUtensorMap mapA,
                                                          const __grid_constant__ CUtensorMap mapB, double* C,
                                                          long long ldc, const double* A, long long lda,
                                                          const double* B, long long ldb, const int* ea,
                                                          const int* eb, int m, int n, int k, int kblocks, int pairs, int mt, int ntiles,
                                                          int* wait_error) {
  pdl_wait();
  pdl_trigger();
  using TL = oz::Tile<BN>;
  constexpr int CW = BN / 2;  // columns per drain warp
  extern __shared__ __align__(1024) unsigned char smem_tiles[];
  unsigned char* tiles = (unsigned char*)(((uintptr_t)smem_tiles + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(tiles + TL::STAGES * TL::STAGE_BYTES);
  uint64_t* empty = full + TL::STAGES;
  uint64_t* acc_full = empty + TL::STAGES;  // [2] MMA -> drain
  uint64_t* acc_empty = acc_full + 2;       // [2] drain -> MMA (8 warp arrivals)
  uint64_t* done = acc_empty + 2;           // all MMAs retired
  uint64_t* decided = done + 1;             // drain -> all: s_more of this tile is final (8 warp arrivals)
  uint32_t* tmem_slot = (uint32_t*)(decided + 1);
  __shared__ int s_fail, s_skip;
  // the last of a CTA's tiles (from 1, by parity) that takes d = 10, d = 11, and
  // d = 10 with the ninth digits
  __shared__ int s_more[3][2];
  // by drain thread and 32 columns: outputs in units of 2^-70, of 2^-78, left to
  // FP64, left to FP64 if they are few
  __shared__ unsigned s_low[(CW + 31) / 32][4][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = CPLX ? 2 * n : n;  // real output columns
  const int kbx = min(oz::KB, kblocks);

  if (threadIdx.x == 0) {
    for (int s = 0; s < TL::STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; a++) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 8); }
    mbar_init(done, 1);
    mbar_init(decided, 8);
    for (int q = 0; q < 6; q++) s_more[q / 2][q % 2] = 0;
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // once a CTA of this call has given up a wait, the rest do no work (read once, so
  // that the whole CTA takes the same way; by a thread with nothing else to do here)
  if (threadIdx.x == 64) s_skip = *(volatile int*)wait_error;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(2 * BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (s_skip) {
  } else if (warp == 0) {
    if (lane == 0) {
      RingPos<TL::STAGES> r;
      int issued = 0;  // stages in use
      bool ok = true;
      for (int t = blockIdx.x, it = 0; t < ntiles && ok; t += gridDim.x, it++) {
        const OzTile tile = oz_tile(t, mt, ntiles);
        const int ya = tile.m * oz::BM, yb = tile.n * BN;
        for (int step = 0; step < oz::STEPS && ok; step++) {
          if (step >= 9) {
            if (step == 9 && !mbar_wait(decided, (uint32_t)(it & 1))) { atomicExch(&s_fail, 1); ok = false; }
            if (!ok || *(volatile int*)&s_more[step - 9][it & 1] != it + 1) break;
          }
          const OzGroup g = oz_group(step, step == 9 && *(volatile int*)&s_more[2][it & 1] != it + 1);
          for (int i = g.i0; i < g.i1 && ok; i++)
            for (int kb = 0; kb < kblocks; kb += kbx, r.next()) {
              // a fresh barrier's previous phase counts as complete
              if (!mbar_wait(&empty[r.s], r.phase ^ 1u)) {
                atomicExch(&s_fail, 1);
                ok = false;
                break;
              }
              unsigned char* sa = tiles + r.s * TL::STAGE_BYTES;
              mbar_arrive_expect_tx(&full[r.s], kbx * (TL::A_BLK + TL::B_BLK));
              tma_load_3d(sa, &mapA, &full[r.s], 0, (i - 1) * m + ya, kb);
              tma_load_3d(sa + TL::A_BYTES, &mapB, &full[r.s], 0, (g.sum - i - 1) * nb + yb, kb);
              issued = min(issued + 1, TL::STAGES);
            }
        }
      }
      // no TMA write may still be in flight when the CTA exits: the last
      // pass of every stage used
      for (int q = 0; q < issued; q++) {
        if (r.s == 0) { r.s = TL::STAGES; r.phase ^= 1u; }
        r.s--;
        mbar_wait(&full[r.s], r.phase);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      RingPos<TL::STAGES> r;
      bool ok = true;
      int u = 0;
      const uint64_t desc0 = sdesc_sw128(smem_u32(tiles));  // addresses count 16 bytes in the low bits
      for (int t = blockIdx.x, it = 0; t < ntiles && ok; t += gridDim.x, it++)
        for (int step = 0; step < oz::STEPS && ok; step++) {
          if (step >= 9) {
            if (step == 9 && !mbar_wait(decided, (uint32_t)(it & 1))) { atomicExch(&s_fail, 1); ok = false; }
            if (!ok || *(volatile int*)&s_more[step - 9][it & 1] != it + 1) break;
          }
          const OzGroup g = oz_group(step, step == 9 && *(volatile int*)&s_more[2][it & 1] != it + 1);
          for (int i0 = g.i0; i0 < g.i1 && ok; i0 += pairs, u++) {
            const int acc = u & 1, i1 = min(i0 + pairs, g.i1);
            if (u >= 2 && !mbar_wait(&acc_empty[acc], (uint32_t)(((u >> 1) - 1) & 1))) {
              atomicExch(&s_fail, 1);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t dt = tmem + (uint32_t)(acc * BN);
            const int steps = (i1 - i0) * ((kblocks + kbx - 1) / kbx);
            for (int st = 0; st < steps; st++, r.next()) {
              if (!mbar_wait(&full[r.s], r.phase)) { atomicExch(&s_fail, 1); ok = false; break; }
              tc_fence_after();
              const uint64_t da = desc0 + (uint32_t)(r.s * (TL::STAGE_BYTES >> 4)), db = da + (TL::A_BYTES >> 4);
#pragma unroll
              for (int kb = 0; kb < oz::KB; kb++) {
                if (kb >= kbx) break;  // (beyond kblocks an odd last box is zero)
#pragma unroll
                for (int kk = 0; kk < oz::BK / 16; kk++)
                  umma_f16(dt, da + kb * (TL::A_BLK >> 4) + 2 * kk, db + kb * (TL::B_BLK >> 4) + 2 * kk, TL::IDESC,
                           (st | kb | kk) ? 1u : 0u);
              }
              umma_commit(&empty[r.s]);
            }
            if (ok) umma_commit(&acc_full[acc]);
          }
        }
      umma_commit(done);
      if (!mbar_wait(done, 0)) atomicExch(&s_fail, 1);
    }
  } else {
    // warp % 4 selects the TMEM lane quarter, the two warps of a quarter
    // split the 128 columns
    const int q = warp & 3, half = (warp - 2) >> 2, dt = threadIdx.x - 64;
    constexpr int CH = 16, NM = (CW + 31) / 32;
    int u = 0;
    bool ok = true;
    for (int t = blockIdx.x, it = 0; t < ntiles && ok; t += gridDim.x, it++) {
      const OzTile tile = oz_tile(t, mt, ntiles);
      const int row = tile.m * oz::BM + q * 32 + lane, col0 = tile.n * BN + half * CW;  // col0: a real column
      unsigned long long T[CW];  // modulo 2^64
      unsigned fine[NM];         // by column: S < S_FINE
      bool some = false;         // outputs of this warp take finer units
#pragma unroll
      for (int h = 0; h < NM; h++) fine[h] = 0;
#pragma unroll
      for (int c = 0; c < CW; c++) T[c] = 0;
      for (int step = 0; step < oz::STEPS && ok; step++) {
        if (step >= 9) {
          if (step == 9) ok = mbar_wait(decided, (uint32_t)(it & 1));
          if (!ok) atomicExch(&s_fail, 1);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok || *(volatile int*)&s_more[step - 9][it & 1] != it + 1) break;
        }
        const OzGroup g = oz_group(step, step == 9 && *(volatile int*)&s_more[2][it & 1] != it + 1);
        // units: 2^-70 for d = 9, 2^-62 down to d = 4, then 2^-53, for a fine
        // output still 2^-62; every sum of the former stays below 2^63.  (Some: 2^-62,
        // 2^-70 or 2^-78 from the first, then 2^-53 for those that are not fine.)
        const int d = g.sum, sh = d >= 8 ? 0 : (d >= 4 ? 8 * (8 - d) : (d == 3 ? 31 : 39)), shf = d <= 3 ? sh + 9 : sh;
        for (int i0 = g.i0; i0 < g.i1; i0 += pairs, u++) {
          const int acc = u & 1;
          ok = mbar_wait(&acc_full[acc], (uint32_t)((u >> 1) & 1));
          if (!ok) atomicExch(&s_fail, 1);
          ok = __all_sync(0xffffffffu, ok && !*(volatile int*)&s_fail);  // the warp together: its TMEM reads are collective
          if (!ok) break;
          tc_fence_after();
          const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * BN + half * CW);
#pragma unroll
          for (int c0 = 0; c0 < CW; c0 += CH) {
            float v[CH];
            tmem_ld16(tb + (uint32_t)c0, v);
            if (c0 + CH == CW) {  // this warp's last read of the buffer
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&acc_empty[acc]);
            }
            if (step == 0) {
              // (a zero sum needs nothing; beyond C's edge they are zero)
              float least = oz::S_FINE;
#pragma unroll
              for (int c = 0; c < CH; c++) {
                if (v[c] < oz::S_FINE) fine[c0 / 32] |= 1u << (c0 + c) % 32;
                least = fminf(least, v[c] > 0.0f ? v[c] : oz::S_FINE);
              }
              unsigned l10 = 0, l11 = 0, l64 = 0, few = 0;
              if (least < oz::S_10) {
#pragma unroll
                for (int c = 0; c < CH; c++) {
                  const unsigned bit = v[c] > 0.0f ? 1u << (c0 + c) % 32 : 0u;
                  if (v[c] < oz::S_10) l10 |= bit;
                  if (v[c] < oz::S_FEW) few |= bit;
                  if (v[c] < oz::S_11) l11 |= bit;
                  if (v[c] < oz::S_FP64) l64 |= bit;
                }
              }
              const int h = c0 / 32;
              if (c0 % 32 == 0) s_low[h][0][dt] = s_low[h][1][dt] = s_low[h][2][dt] = s_low[h][3][dt] = 0;
              if (l10) {
                s_low[h][0][dt] |= l10;
                s_low[h][1][dt] |= l11;
                s_low[h][2][dt] |= l64;
                s_low[h][3][dt] |= few;
              }
            } else if (some) {
              const unsigned l10 = s_low[c0 / 32][0][dt], l11 = s_low[c0 / 32][1][dt];
#pragma unroll
              for (int c = 0; c < CH; c++) {
                const int bit = (c0 + c) % 32;
                const bool f = (fine[c0 / 32] >> bit) & 1;
                // 2^-(8d - 2) in units of 2^-62, 2^-70 or 2^-78 (or 2^-53)
                const int r = 64 - 8 * d + (((l10 >> bit) & 1) << 3) + (((l11 >> bit) & 1) << 3) - (d <= 3 && !f ? 9 : 0);
                const long long x = (long long)__float2int_rn(v[c]);
                const unsigned long long y = r >= 0 ? shl64(x, r) : (unsigned long long)((x + (1ll << (-r - 1))) >> -r);
                if (d < 10 || f) T[c0 + c] += y;
              }
            } else if (step == 9) {
#pragma unroll
              for (int c = 0; c < CH; c++)
                if ((fine[c0 / 32] >> (c0 + c) % 32) & 1) T[c0 + c] += (unsigned long long)(long long)((__float2int_rn(v[c]) + (1 << 15)) >> 16);
            } else if (step == 10) {
              // nothing of d = 11 counts here
            } else if (sh == shf) {
#pragma unroll
              for (int c = 0; c < CH; c++) T[c0 + c] += (unsigned long long)(long long)__float2int_rn(v[c]) << sh;
            } else {
#pragma unroll
              for (int c = 0; c < CH; c++)
                T[c0 + c] += (unsigned long long)(long long)__float2int_rn(v[c]) << (((fine[c0 / 32] >> (c0 + c) % 32) & 1) ? shf : sh);
            }
          }
        }
        if (!ok) break;
        if (step == 0) {
          // how small the warp's outputs are: d = 10 for some; beyond FEW below
          // S_FEW, finer units too
          unsigned any10 = 0, any11 = 0, nfew = 0;
#pragma unroll
          for (int h = 0; h < NM; h++) {
            any10 |= s_low[h][0][dt];
            any11 |= s_low[h][1][dt];
            nfew += __popc(s_low[h][3][dt]);
          }
          some = __reduce_add_sync(0xffffffffu, nfew) > oz::FEW;
          any10 = __any_sync(0xffffffffu, any10 != 0);
          any11 = __any_sync(0xffffffffu, any11 != 0);
          if (!some) {
#pragma unroll
            for (int h = 0; h < NM; h++) {
              s_low[h][0][dt] = s_low[h][1][dt] = 0;
              s_low[h][2][dt] = s_low[h][3][dt];
            }
          }
          if (lane == 0) {
            if (any10) atomicMax(&s_more[0][it & 1], it + 1);
            if (some && any11) atomicMax(&s_more[1][it & 1], it + 1);
            if (some) atomicMax(&s_more[2][it & 1], it + 1);
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(decided);
        }
        if (d == 9 && !some) {
#pragma unroll
          for (int c = 0; c < CW; c++) T[c] = (unsigned long long)(((long long)T[c] + 128) >> 8);
        }
        if (d == 4) {
#pragma unroll
          for (int c = 0; c < CW; c++)
            if (!((fine[c / 32] >> (c % 32)) & 1)) T[c] = (unsigned long long)(((long long)T[c] + 256) >> 9);
        }
      }
      if (!ok) break;
      constexpr int W = CPLX ? 2 : 1;
      const int j0 = col0 / W;
      unsigned l10[NM], l11[NM], l64[NM];
#pragma unroll
      for (int h = 0; h < NM; h++) {
        l10[h] = s_low[h][0][dt];
        l11[h] = s_low[h][1][dt];
        l64[h] = s_low[h][2][dt];
      }
      if (row < m) {
        const int er = ea[row];
        constexpr int EB = 4;  // C's elements in flight: their loads are a trip to memory each
#pragma unroll
        for (int cb = 0; cb < CW; cb += EB * W) {
          double z[EB][W];
          int ec[EB];
#pragma unroll
          for (int b = 0; b < EB; b++) {
            const int j = min(j0 + cb / W + b, n - 1);
            const double* p = C + W * ((long long)row + (long long)j * ldc);
            ec[b] = eb[j];
            if (CPLX) {
              const double2 zz = *reinterpret_cast<const double2*>(p);
              z[b][0] = zz.x; z[b][W - 1] = zz.y;
            } else {
              z[b][0] = *p;
            }
          }
#pragma unroll
          for (int b = 0; b < EB; b++) {
            const int c = cb + b * W, j = j0 + c / W, e = er + ec[b] - 53;
            // the unit of the sum, 2^-53 less 0, 9, 17 or 25
            auto unit = [&](int cc) {
              const int h = cc / 32, bit = cc % 32;
              return e - (((fine[h] >> bit) & 1) * 9 + ((((l10[h] >> bit) & 1) + ((l11[h] >> bit) & 1)) << 3));
            };
#pragma unroll
            for (int w = 0; w < W; w++) z[b][w] -= int_to_double((long long)T[c + w], unit(c + w));
            if (j < n && !((l64[c / 32] >> (c % 32)) & (W == 2 ? 3u : 1u))) {
              double* p = C + W * ((long long)row + (long long)j * ldc);
              if (CPLX) *reinterpret_cast<double2*>(p) = make_double2(z[b][0], z[b][W - 1]);
              else *p = z[b][0];
            }
          }
        }
      }
#pragma unroll
      for (int h = 0; h < NM; h++)
        if (__any_sync(0xffffffffu, l64[h] != 0)) oz_fp64<CPLX>(C, ldc, A, lda, B, ldb, m, n, k, row, j0 + h * 32 / W, l64[h]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN));
  }
  if (threadIdx.x == 0 && s_fail) atomicExch(wait_error, 1);
}

static size_t oz_round(size_t x) { return (x + 1023) & ~(size_t)1023; }

size_t oz_gemm_ws_bytes(int m, int n, int k, bool cplx) {
  const size_t Kp = ((size_t)(cplx ? 2 * k : k) + 63) / 64 * 64, nb = cplx ? 2 * (size_t)n : (size_t)n;
  return oz_round((oz::NS + 1) * (size_t)m * Kp * 2) + oz_round((oz::NS + 1) * nb * Kp * 2) + oz_round(4 * (size_t)m) +
         oz_round(4 * (size_t)n) + 1024;
}

// false (and *err = cudaSuccess): not taken -- more products per output than
// the accumulators add exactly, or too little workspace; the caller's SIMT
// update does it
template <bool CPLX>
static bool update(double* C, long long ldc, const double* A, long long lda, const double* B, long long ldb, int m,
                   int n, int k, void* ws, size_t ws_bytes, int* wait_error, cudaStream_t s, cudaError_t* err) {
  *err = cudaSuccess;
  if (!tensor_updates()) return false;  // GBEM_LU_TC=0
  if (m <= 0 || n <= 0 || k <= 0) return true;
  const int kreal = CPLX ? 2 * k : k;
  if (kreal > oz::KMAX || !ws || ws_bytes < oz_gemm_ws_bytes(m, n, k, CPLX)) return false;
  const int Kp = (kreal + 63) / 64 * 64, nb = CPLX ? 2 * n : n;
  unsigned char* w = (unsigned char*)(((uintptr_t)ws + 1023) & ~(uintptr_t)1023);
  __nv_bfloat16* pa = (__nv_bfloat16*)w; w += oz_round((oz::NS + 1) * (size_t)m * Kp * 2);
  __nv_bfloat16* pb = (__nv_bfloat16*)w; w += oz_round((oz::NS + 1) * (size_t)nb * Kp * 2);
  int* ea = (int*)w; w += oz_round(4 * (size_t)m);
  int* eb = (int*)w;
  const int na = (m + oz::VECS - 1) / oz::VECS, nbk = (n + oz::VECS - 1) / oz::VECS;
  if ((*err = allow_max_smem(oz_pack<CPLX>)) != cudaSuccess) return false;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int mt = (m + oz::BM - 1) / oz::BM;
  // narrow tiles where one wave of them covers C: a tile's k-steps and drain
  // are then shorter (m = 3584, n = k = 32, seven digits: 23 us with packing, 35 with
  // 128 columns); in two waves they lose (m = n = 704, k = 256: 170 against 113)
  const int bn = mt * ((nb + 31) / 32) <= nsm ? 32 : 128;
  const auto kernel = bn == 32 ? oz_gemm_kernel<CPLX, 32> : oz_gemm_kernel<CPLX, 128>;
  const int smem = bn == 32 ? oz::Tile<32>::SMEM_BYTES : oz::Tile<128>::SMEM_BYTES;
  if ((*err = allow_max_smem(kernel)) != cudaSuccess) return false;
  CUtensorMap ma, mb;
  if (!make_bf16_map(&ma, pa, (oz::NS + 1LL) * m, Kp, oz::BM, std::min(oz::KB, Kp / oz::BK)) ||
      !make_bf16_map(&mb, pb, (oz::NS + 1LL) * nb, Kp, bn, std::min(oz::KB, Kp / oz::BK)))
    return false;
  *err = launch_pdl(oz_pack<CPLX>, dim3(na + nbk), dim3(256), (size_t)k * 17 * (CPLX ? 16 : 8), s, A, lda, m, B, ldb, n,
                    k, Kp, na, pa, pb, ea, eb);
  if (*err != cudaSuccess) return false;
  const int ntiles = mt * ((nb + bn - 1) / bn);
  *err = launch_pdl(kernel, dim3(std::min(ntiles, nsm)), dim3(320), (size_t)smem, s, ma, mb, C, ldc, A, lda, B, ldb, ea, eb, m, n, k,
                    Kp / oz::BK, oz::ACC_TERMS / kreal, mt, ntiles, wait_error);
  return *err == cudaSuccess;
}

bool oz_gemm_update(cx<double>* C, long long ldc, const cx<double>* A, long long lda, const cx<double>* B, long long ldb,
                    int m, int n, int k, void* ws, size_t ws_bytes, int* wait_error, cudaStream_t s, cudaError_t* err) {
  return update<true>((double*)C, ldc, (const double*)A, lda, (const double*)B, ldb, m, n, k, ws, ws_bytes, wait_error, s, err);
}
bool oz_gemm_update(double* C, long long ldc, const double* A, long long lda, const double* B, long long ldb, int m,
                    int n, int k, void* ws, size_t ws_bytes, int* wait_error, cudaStream_t s, cudaError_t* err) {
  return update<false>(C, ldc, A, lda, B, ldb, m, n, k, ws, ws_bytes, wait_error, s, err);
}

}  // namespace gbem
