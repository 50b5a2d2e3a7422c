// gemm_oz.cu -- the FP64 matrix update on the tensor cores:
//     C (m x n) -= A (m x k) * B (k x n)
// for complex128 or real double, column-major, to FP64 accuracy, with
// tcgen05.mma (kind::f16) on integer slices of the operands (the error-free
// splitting of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication and
// its applications", Numer. Algorithms 59, 2012).
//
// Each row of A and each column of B is scaled by the power of two above its
// largest entry and rounded to a 55-bit fixed-point number, written as seven
// balanced base-256 digits (-128 .. 128, exact in bf16).  The product of two
// digit matrices is an integer; its FP32 accumulator is exact while it stays
// within 2^24, that is over 1024 products of at most 2^14.  The pairs (i, j)
// of slices with i + j = d share the weight 2^-(8d - 2), so they add up in one
// accumulator, as many pairs as the 1024 products allow; the groups d = 2 .. 9
// (34 of the 49 pairs) are drained into one 64-bit integer per output, which
// is rounded to FP64 once (integer arithmetic) and subtracted from C.  What is
// left is the rounding to 55 bits, 2^-56 of the row's or column's maximum per
// entry: for a row of L with entries below 1 and a column of U about
// 2^-53 * 0.24 sqrt(k) of the column's typical entry, an FP64 chain's
// 2^-53 * 0.3 sqrt(k).  (Without d = 9 it is three times that: the backward
// error of an LU of normal entries, N = 768, was 1.06e-14 against 5.6e-15 for
// FP64 chains.)
//
// Measured, k = 256: 30 TFLOP/s FP64 at m = n = 15104 (1000 TFLOP/s of bf16,
// 55 % of the measured rate) against 0.74 for the SIMT FP64 update; the
// updates of an N = 3840 LU 6 ms against 194.  Error against long double for
// normal entries, k = 256: 4.9e-18 of |a| |b| root mean square, FP64 FMAs
// 4.3e-17; backward error of an LU of normal entries, N = 768: 3.3e-15 against
// 5.6e-15 with FP64 updates (LAPACK 6.3e-15).
//
// What bounds it: the instructions of the single-thread TMA and MMA issuers
// per k-step at every size, and the tensor pipe (34 bf16 products in place of
// one FP64 one) not far behind.  The FP64 pipe it replaces runs 2 FMAs per
// cycle and SM.
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
constexpr int NS = 7;             // slices (base-256 digits)
constexpr int DMAX = 9;           // largest i + j of the slice pairs taken
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
  static_assert((2 * STAGES + 5) * 8 + 4 <= 256, "barrier area");
  static_assert(B_BLK % 1024 == 0, "swizzle atoms");
};
constexpr int EXP_BAD = 1 << 20;  // scale exponent of a row or column that is not finite
constexpr int VECS = 16;          // rows of A (columns of B) per packing CTA
}  // namespace oz

// exponent field (at least 1) of a double's high word
__device__ __forceinline__ int exp_field(unsigned hi) { return max((int)((hi >> 20) & 0x7ffu), 1); }

// |x| < 2^(F - 1022) as a signed 55-bit fixed-point number: round(x 2^(55 - (F - 1022)))
__device__ __forceinline__ long long fixed55(double x, int F) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int raw = (int)((b >> 52) & 0x7ffu), f = max(raw, 1);
  unsigned long long M = b & 0xfffffffffffffull;
  if (raw) M |= 1ull << 52;
  const int d = F - f;  // >= 0
  unsigned long long q;
  if (d <= 2) q = M << (2 - d);
  else if (d < 58) q = (M + (1ull << (d - 3))) >> (d - 2);
  else q = 0;
  return (long long)b < 0 ? -(long long)q : (long long)q;
}

// The digits of A's rows (part 0) and B's columns (part 1), one launch: CTAs
// [0, na) take 16 rows of A each, the others 16 columns of B.  The vectors
// are staged in shared memory (coalesced), their largest exponent is found,
// and each vector's digits are written slice by slice, out[s][row][Kp],
// zero beyond kreal.  A complex row of A is [Re | Im]; a complex column j of
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
    long long b[4];  // bytes 0..5: digits 7..2 plus 128; above: the top digit
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
      b[e] = (F < 0 ? 0 : fixed55(x, F)) + 0x808080808080ll;
    }
#pragma unroll
    for (int s = 0; s < oz::NS; s++) {  // slice s holds digit s + 1 (the top one first)
      unsigned short w[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const int dg = s == 0 ? (int)(b[e] >> 48) : (int)((b[e] >> (8 * (6 - s))) & 255) - 128;
        w[e] = (unsigned short)(__float_as_uint((float)((neg >> e) & 1u ? -dg : dg)) >> 16);
      }
      uint2 pk;
      pk.x = (unsigned)w[0] | ((unsigned)w[1] << 16);
      pk.y = (unsigned)w[2] | ((unsigned)w[3] << 16);
      *reinterpret_cast<uint2*>(out + ((long long)s * rows + (long long)v0 * rpv + r) * Kp + 4 * g) = pk;
    }
  }
}

// T 2^e rounded to 53 bits, -1000 < e < 960, in integer arithmetic: the FP64
// pipe (2 operations per cycle and SM) is left with the one subtraction.
__device__ __forceinline__ double int_to_double(long long T, int e) {
  const unsigned long long a = T < 0 ? 0ull - (unsigned long long)T : (unsigned long long)T;
  const int lz = __clzll((long long)a);
  const unsigned long long m = a << (lz & 63);
  const unsigned long long q = (m >> 11) + ((m >> 10) & 1ull);  // 2^52 .. 2^53
  unsigned long long b = ((unsigned long long)(1023 + 63 - 1 + e - lz) << 52) + q;
  b |= (unsigned long long)T & 0x8000000000000000ull;
  return a ? __longlong_as_double((long long)b) : 0.0;
}

// One CTA per SM walks the 128 x BN output tiles (columns counted as reals;
// m fastest, so the CTAs of a wave share their B tile).  Warp 0: TMA producer;
// warp 1: TMEM and MMA issue; warps 2-9: drain.  A tile's accumulators follow
// one another through two BN-column TMEM buffers: the MMAs of the next run
// while the drain warps add the last one into their 64-bit integers (one row
// and BN / 2 columns per thread).  pairs: slice pairs per accumulator.
template <bool CPLX, int BN>
__global__ void __launch_bounds__(320, 1) oz_gemm_kernel(const __grid_constant__ CUtensorMap mapA,
                                                          const __grid_constant__ CUtensorMap mapB, double* C,
                                                          long long ldc, const int* ea, const int* eb, int m, int n,
                                                          int kblocks, int pairs, int mt, int ntiles,
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
  uint32_t* tmem_slot = (uint32_t*)(done + 1);
  __shared__ int s_fail, s_skip;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = CPLX ? 2 * n : n;  // real output columns
  const int kbx = min(oz::KB, kblocks);

  if (threadIdx.x == 0) {
    for (int s = 0; s < TL::STAGES; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; a++) { mbar_init(&acc_full[a], 1); mbar_init(&acc_empty[a], 8); }
    mbar_init(done, 1);
    s_fail = 0;
    // once a CTA of this call has given up a wait, the rest do no work (read
    // once, so that the whole CTA takes the same way)
    s_skip = *(volatile int*)wait_error;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
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
      for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
        const int ya = (t % mt) * oz::BM, yb = (t / mt) * BN;
        for (int d = oz::DMAX; d >= 2 && ok; d--)
          for (int i = max(1, d - oz::NS); i <= min(oz::NS, d - 1) && ok; i++)
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
              tma_load_3d(sa + TL::A_BYTES, &mapB, &full[r.s], 0, (d - i - 1) * nb + yb, kb);
              issued = min(issued + 1, TL::STAGES);
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
      for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x)
        for (int d = oz::DMAX; d >= 2 && ok; d--) {
          const int ie = min(oz::NS + 1, d);
          for (int i0 = max(1, d - oz::NS); i0 < ie && ok; i0 += pairs, u++) {
            const int acc = u & 1, i1 = min(i0 + pairs, ie);
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
    const int q = warp & 3, half = (warp - 2) >> 2;
    constexpr int CH = CW < 32 ? CW : 32;
    int u = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
      const int tm = t % mt, tn = t / mt;
      const int row = tm * oz::BM + q * 32 + lane;
      long long T[CW];
#pragma unroll
      for (int c = 0; c < CW; c++) T[c] = 0;
      for (int d = oz::DMAX; d >= 2 && ok; d--) {
        // units 2^-70 for d = 9, 2^-62 down to d = 4, then 2^-53: every sum
        // stays below 2^63
        const int sh = d >= 8 ? 0 : (d >= 4 ? 8 * (8 - d) : (d == 3 ? 31 : 39));
        const int ie = min(oz::NS + 1, d);
        for (int i0 = max(1, d - oz::NS); i0 < ie; i0 += pairs, u++) {
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
            if constexpr (CH == 32) tmem_ld32(tb + (uint32_t)c0, v);
            else tmem_ld16(tb + (uint32_t)c0, v);
            if (c0 + CH == CW) {  // this warp's last read of the buffer
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&acc_empty[acc]);
            }
#pragma unroll
            for (int c = 0; c < CH; c++) T[c0 + c] += (long long)__float2int_rn(v[c]) << sh;
          }
        }
        if (d == 9 || d == 4) {
          const int down = d == 9 ? 8 : 9;
#pragma unroll
          for (int c = 0; c < CW; c++) T[c] = (T[c] + (1 << (down - 1))) >> down;
        }
      }
      if (!ok) break;
      if (row < m) {
        const int er = ea[row];
        constexpr int W = CPLX ? 2 : 1;
        const int j0 = (tn * BN + half * CW) / W;
#pragma unroll
        for (int c = 0; c < CW; c += W) {
          const int j = j0 + c / W;
          if (j >= n) break;
          const int ec = eb[j], e = er + ec - 53;
          double* p = C + W * ((long long)row + (long long)j * ldc);
          double z[W];
          if (CPLX) {
            const double2 zz = *reinterpret_cast<const double2*>(p);
            z[0] = zz.x; z[W - 1] = zz.y;
          } else {
            z[0] = *p;
          }
          if (e > -1000 && e < 960) {
#pragma unroll
            for (int w = 0; w < W; w++) z[w] -= int_to_double(T[c + w], e);
          } else if (er == oz::EXP_BAD || ec == oz::EXP_BAD) {
#pragma unroll
            for (int w = 0; w < W; w++) z[w] = __longlong_as_double(0x7ff8000000000000ll);
          } else {
#pragma unroll
            for (int w = 0; w < W; w++) z[w] -= ldexp((double)T[c + w], e);
          }
          if (CPLX) *reinterpret_cast<double2*>(p) = make_double2(z[0], z[W - 1]);
          else *p = z[0];
        }
      }
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
  return oz_round(oz::NS * (size_t)m * Kp * 2) + oz_round(oz::NS * nb * Kp * 2) + oz_round(4 * (size_t)m) +
         oz_round(4 * (size_t)n) + 1024;
}

// false (and *err = cudaSuccess): not taken -- more products per output than
// the accumulators add exactly, or too little workspace; the caller's SIMT
// update does it
template <bool CPLX>
static bool update(double* C, long long ldc, const double* A, long long lda, const double* B, long long ldb, int m,
                   int n, int k, void* ws, size_t ws_bytes, int* wait_error, cudaStream_t s, cudaError_t* err) {
  *err = cudaSuccess;
  if (m <= 0 || n <= 0 || k <= 0) return true;
  const int kreal = CPLX ? 2 * k : k;
  if (kreal > oz::KMAX || !ws || ws_bytes < oz_gemm_ws_bytes(m, n, k, CPLX)) return false;
  const int Kp = (kreal + 63) / 64 * 64, nb = CPLX ? 2 * n : n;
  unsigned char* w = (unsigned char*)(((uintptr_t)ws + 1023) & ~(uintptr_t)1023);
  __nv_bfloat16* pa = (__nv_bfloat16*)w; w += oz_round(oz::NS * (size_t)m * Kp * 2);
  __nv_bfloat16* pb = (__nv_bfloat16*)w; w += oz_round(oz::NS * (size_t)nb * Kp * 2);
  int* ea = (int*)w; w += oz_round(4 * (size_t)m);
  int* eb = (int*)w;
  const int na = (m + oz::VECS - 1) / oz::VECS, nbk = (n + oz::VECS - 1) / oz::VECS;
  if ((*err = allow_max_smem(oz_pack<CPLX>)) != cudaSuccess) return false;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int mt = (m + oz::BM - 1) / oz::BM;
  // narrow tiles where one wave of them covers C: a tile's k-steps and drain
  // are then shorter (m = 3584, n = k = 32: 23 us with packing, 35 with
  // 128 columns); in two waves they lose (m = n = 704, k = 256: 170 against 113)
  const int bn = mt * ((nb + 31) / 32) <= nsm ? 32 : 128;
  const auto kernel = bn == 32 ? oz_gemm_kernel<CPLX, 32> : oz_gemm_kernel<CPLX, 128>;
  const int smem = bn == 32 ? oz::Tile<32>::SMEM_BYTES : oz::Tile<128>::SMEM_BYTES;
  if ((*err = allow_max_smem(kernel)) != cudaSuccess) return false;
  CUtensorMap ma, mb;
  if (!make_bf16_map(&ma, pa, (long long)oz::NS * m, Kp, oz::BM, std::min(oz::KB, Kp / oz::BK)) ||
      !make_bf16_map(&mb, pb, (long long)oz::NS * nb, Kp, bn, std::min(oz::KB, Kp / oz::BK)))
    return false;
  *err = launch_pdl(oz_pack<CPLX>, dim3(na + nbk), dim3(256), (size_t)k * 17 * (CPLX ? 16 : 8), s, A, lda, m, B, ldb, n,
                    k, Kp, na, pa, pb, ea, eb);
  if (*err != cudaSuccess) return false;
  const int ntiles = mt * ((nb + bn - 1) / bn);
  *err = launch_pdl(kernel, dim3(std::min(ntiles, nsm)), dim3(320), (size_t)smem, s, ma, mb, C, ldc, ea, eb, m, n,
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
