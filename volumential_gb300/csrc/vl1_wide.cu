// FP64-accurate list-1 evaluation on the tensor cores (tcgen05, 8 + 8 FP16
// digits, exact partial products, integer sums, one rounding to FP64).
//
// The FP64 pipe of this GPU (about 1.1 TFLOP/s) bounds the plain kernel: a 3D
// q = 4 tree of 1.5M points and 2.3e9 point pairs takes 4.7 ms at 0.98
// TFLOP/s.  Here the same sums are formed from digit products, as in the
// mixed path (vl1_mixed.cu), but with so many digits that a box's results are
// as accurate as FP64 sums against the largest product of its list:
//
//   x' = scaling * coefficient = 2^(E + 1) sum_{i=1..8} X_i 2^(-8i)
//   T                          = 2^(A + 1) sum_{j=1..8} T_j 2^(-8j)
//
// with balanced base-256 digits (|digit| <= 128, |X_1| <= 512, exact in
// FP16).  E is the exponent of the largest |x'| of the *density row* (source
// box, rhs), less 2, rounded up to a multiple of 8 (the leading digit takes
// two more bits, so that at most 5 of the 63 are lost to the rounding), and A
// that of the table block (table level, case), equal to the largest block's
// modulo 8.  A target row sums sources of different E + A: with all of them
// equal modulo 8 the sum against the largest one is a shift by whole digits,
// so the producers only read each source's digit planes from an offset
// (position p takes plane p - (E_t - E - A) / 8, zero above).  Every target
// box thus has its own scale, the largest E + A of the pairs it sums, whatever
// the range of the density over the domain and of the blocks over the table.
//
// The products i + j = d of weight 2^(-8d) share an accumulator: d = 2..6 are
// exact integers over a round of 128 source points (at most
// 128 * (2^16 + 4 * 2^14) = 2^24 in FP32) and are read out after every round
// into an int64; d = 7..9 accumulate in FP32 over the whole work item.  Their
// digits are balanced and, past the leading ones, without a sign of their
// own, so their sums stay near 2^20, where FP32 is exact too; sums beyond
// 2^24 need products of one sign throughout, leading digits included, and
// then the rounding of d = 7 is below 2^-53 of the result.  d >= 10 is dropped
// (2^-66 per pair in the mean square).  The result is rounded once.  Against
// 113-bit sums (2D and 3D, q = 1..16, Laplace- and Helmholtz-like tables, real
// and complex densities, densities over 6 and 200 decades) the relative l2
// error is 4e-17 .. 2e-16, the per-box kernel's 1e-16 .. 2e-15.
//
// The error is against max|x'| max|T| over a row's pairs, not against each
// target's own products: with K source points at most 6 * 2^-50.2 sqrt(K) of
// that maximum where the roundings of E and A to multiples of 8 fall worst
// (test_gpu_fp64_digits.py), some 2^-60 where they fall well.  A target whose
// products all lie far below it keeps fewer bits than an FP64 sum: with one
// source point in the corner neighbour up to 1e-15 (3D, q = 4) and 5e-15 (2D,
// q = 6) of its value, 1e-16 per box.
//
// Measured (GB300, a call's device time): the 1.5M-point octree 4,610 us
// per-box, 232 us here (digits and the comparison of the tree's arrays about 24
// us, tensor-core kernel 206 us, its tensor pipe busy 105 us of them); 3D q = 5,
// 512,000 points 3,220 and 169 us; 3D q = 3, 110,592 points x 8 right-hand sides
// 1,400 and 127 us; 2D complex q = 5, 102,400 points 174 and 43 us.  Bound:
// shared memory (per unit 120 KB of operand reads and 48 KB of stores, 1,350 of
// the ~1,750 clocks) and the L2's delivery to all SMs (36 KB at ~30 bytes per SM
// and clock, 1,200), close behind them the tensor pipe (1,176); per work item
// ~12 us of start and result write.
//
// Density rows with an infinite or NaN value (or whose scaled value
// overflows) cannot be written in fixed point: every target row with such a
// source is summed in FP64 by the CTA that writes its tile.
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>

#include "vl1_internal.cuh"
#include "vl1_pipe.cuh"
#include "vl1_tc.cuh"
#include "vl1_wide.cuh"

namespace vl1 {

extern uint32_t g_test_wait_limit_us;   // vl1_test_set_wait_fault
extern int32_t g_test_withhold;

namespace {

constexpr int kW = 8;                 // digits of each operand
constexpr int kWideBits = 8 * kW - 1; // magnitude bits below the exponent
constexpr int kTopBits = 2;           // the density rows' extra leading bits
constexpr int kUnitK = 16;            // source points per pipeline unit
constexpr int kRoundUnits = 8;        // units per exact round (128 source points)
constexpr int kRowUnitBytes = 160;     // a density row's digits of one unit
constexpr int kZeroExp = -100000;     // exponent of an all-zero row or block
constexpr int kBadExp = 1 << 28;      // row with a non-finite value

// The kW balanced digits of |v| < 2^(e + kTopBits) against 2^e, most
// significant first, without the sign: |v| 2^(kWideBits - e) rounded to
// nearest, its low byte and the rest (57 bits and kTopBits) apart.  Adding
// 128 to every byte but the top one makes the additions' carries do the digit
// borrows: a byte b with a carry in becomes b + carry - 256, with a carry
// out, exactly when that is at least 128 - so a digit is its byte minus 128.
struct WideDigits {
  unsigned long long hi;   // biased bytes of digits 0 (all above bit 48) .. 6
  unsigned lo;             // biased byte of digit 7
};
__device__ __forceinline__ WideDigits wide_digits(double v, int e) {
  const unsigned long long mag =
      static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7FFFFFFFFFFFFFFFull;
  const int ef = (int)(mag >> 52);
  const unsigned long long M = ef ? ((mag & 0xFFFFFFFFFFFFFull) | (1ull << 52)) : mag;
  const int sh = (ef ? ef - 1075 : -1074) + kWideBits - e;
  unsigned long long hi;
  unsigned lo;
  if (sh >= 8) {          // sh <= 10 + kTopBits for M of 53 bits
    hi = sh < 64 ? M << (sh - 8) : 0ull;
    lo = 0u;
  } else {
    unsigned long long m;
    if (sh >= 0) {        // M < 2^53: fits
      m = M << sh;
    } else {
      const int k = -sh;
      m = k > 54 ? 0ull : (M + ((1ull << (k - 1)) - 1ull) + ((M >> k) & 1ull)) >> k;
    }
    hi = m >> 8;
    lo = (unsigned)m & 0xFFu;
  }
  WideDigits d;
  lo += 0x80u;
  d.lo = lo & 0xFFu;
  d.hi = hi + (lo >> 8) + 0x0000808080808080ull;
  return d;
}
__device__ __forceinline__ int wide_digit(const WideDigits &d, int i, int sgn) {
  if (i == 0) return sgn * (int)(d.hi >> 48);
  if (i == kW - 1) return sgn * ((int)d.lo - 128);
  return sgn * ((int)((d.hi >> (8 * (kW - 2 - i))) & 0xFFull) - 128);
}

// ----------------------------------------------------- plan: table digits

// exponent of every (table level, case) block: the smallest A >= the block's
// own exponent that equals a_max modulo 8 (kZeroExp for a zero block)
__global__ void wide_key_exp_kernel(DevDesc d, int a_max, int *key_exp) {
  const int key = blockIdx.x;
  const int64_t n = (int64_t)d.nq * d.nq * (d.table_cplx ? 2 : 1);
  const double *B = d.blocks + (int64_t)key * n;
  int e = kZeroExp;
  for (int64_t i = threadIdx.x; i < n; i += blockDim.x) {
    const double v = B[i];
    if (v != 0.0) e = max(e, scale_exponent(v));
  }
  __shared__ int s_e;
  if (threadIdx.x == 0) s_e = kZeroExp;
  __syncthreads();
  if (e != kZeroExp) atomicMax(&s_e, e);
  __syncthreads();
  if (threadIdx.x == 0)
    key_exp[key] = s_e == kZeroExp ? kZeroExp : a_max - 8 * ((a_max - s_e) / 8);
}

// digits of the blocks: [key][unit][column chunk][digit][nch][16] FP16 in the
// swizzled K-major order of shared memory, so that one pipeline unit of one
// chunk is one contiguous bulk copy.  Complex tables: column 2t (2t + 1) is
// the real (imaginary) part of target point t.
__global__ void wide_digits_kernel(DevDesc d, WideGeom g, const int *key_exp, __half *adig) {
  const int64_t per_tile = (int64_t)g.nch * kUnitK;
  const int n_chunks = g.np / g.nch, n_units = g.kp / kUnitK;
  const int64_t n = (int64_t)d.n_tables * d.n_cases * n_units * n_chunks * per_tile;
  const int cv = d.table_cplx ? 2 : 1;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < n;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t rem = idx % per_tile;
    const int col = (int)(rem / kUnitK), k = (int)(rem % kUnitK);
    const int64_t tile = idx / per_tile;            // (key, unit, chunk)
    const int chunk = (int)(tile % n_chunks);
    const int64_t ku = tile / n_chunks;
    const int s = (int)(ku % n_units) * kUnitK + k;
    const int key = (int)(ku / n_units);
    const int n_col = chunk * g.nch + col;
    const int t = n_col / cv, part = n_col - t * cv;
    double v = 0.0;
    if (s < d.nq && t < d.nq)
      v = d.blocks[(((int64_t)key * d.nq + s) * d.nq + t) * cv + part];
    const int e = key_exp[key];
    const WideDigits bd = e == kZeroExp ? wide_digits(0.0, 0) : wide_digits(v, e);
    const int sgn = __double_as_longlong(v) < 0 ? -1 : 1;
    const uint32_t off = tc::kmajor_swizzled_offset(col, k, kUnitK) / 2;
#pragma unroll
    for (int i = 0; i < kW; ++i)
      adig[(tile * kW + i) * per_tile + off] = __int2half_rn(wide_digit(bd, i, sgn));
  }
}

// ------------------------------------------------- per call: density rows

// Digits of a density value against 2^e for storage as bytes: the signed
// fixed-point number in two's complement, so that a digit is its byte minus
// 128 (-128 .. 127) with the sign included, and only the leading one
// (-512 .. 512) is wider.
struct RowDigits {
  long long hi;   // leading digit << 48 | biased bytes of digits 1..6
  unsigned lo;    // biased byte of digit 7
};
__device__ __forceinline__ RowDigits row_digits(double v, int e) {
  const WideDigits m = wide_digits(fabs(v), e);   // biased: take the bias out again
  unsigned lo = (m.lo + 0x80u) & 0xFFu;           // low byte of the magnitude
  long long hi = (long long)(m.hi - (unsigned long long)(m.lo < 0x80u ? 1 : 0) -
                             0x0000808080808080ull);
  if (v < 0.0) {
    hi = -hi - (lo != 0u ? 1 : 0);
    lo = (0u - lo) & 0xFFu;
  }
  lo += 0x80u;
  RowDigits d;
  d.lo = lo & 0xFFu;
  d.hi = hi + (long long)(lo >> 8) + 0x0000808080808080ll;
  return d;
}

// a tree array now and when the schedule was made
struct Span {
  const uint8_t *now, *then;
  int64_t bytes, chunks;   // chunks: of 16 bytes, 0 for an array at an odd address
};
constexpr int kSpans = 8;

// A density row is (source box b, virtual rhs v), row index b * nv + v.  Real
// coefficients: v is the rhs.  Complex coefficients: v = 2 * rhs + part.
struct WidePrep {
  DevDesc d;
  TreeDev tr;
  const double *coefs;
  int cc;            // complex coefficients
  int nv;
  int kp;
  int *x_exp;        // per row: exponent (a multiple of 8), kZeroExp or kBadExp
  double *wbox;      // per row: the 2D log displacement's sum over the box (nullptr: none)
  uint8_t *xpl;      // digits [row][unit][160 bytes], see wide_prep_kernel
  int *counters;     // split counters, zeroed here
  int n_counters;
  Span spans[kSpans];
  int64_t max_chunks;
  int row_blocks;    // blocks that form digits; the others compare the arrays
  int *stale;        // nullptr: the caller answers for the schedule
  vl1_status *st;
};

// Whether the arrays differ from those that the schedule was made from.  A
// schedule outlives the call that made it, and its arrays' owner may write them
// by ways that leave no trace on the host (a kernel, a graph's replay): every
// call compares them, 16 bytes of every array at a time so that the loads are
// in flight together (10 MB each on the 1.5M-point octree).
__device__ __forceinline__ bool tree_differs(const WidePrep &P, int64_t i0, int64_t n) {
  unsigned acc = 0u;
  for (int64_t c = i0; c < P.max_chunks; c += n) {
#pragma unroll
    for (int k = 0; k < kSpans; ++k) {
      if (c >= P.spans[k].chunks) continue;
      const uint4 x = __ldg(reinterpret_cast<const uint4 *>(P.spans[k].now) + c);
      const uint4 y = __ldg(reinterpret_cast<const uint4 *>(P.spans[k].then) + c);
      acc |= (x.x ^ y.x) | (x.y ^ y.y) | (x.z ^ y.z) | (x.w ^ y.w);
    }
  }
#pragma unroll 1
  for (int k = 0; k < kSpans; ++k)   // the last bytes, and arrays at odd addresses
    for (int64_t b = P.spans[k].chunks * 16 + i0; b < P.spans[k].bytes; b += n)
      acc |= (unsigned)(P.spans[k].now[b] ^ P.spans[k].then[b]);
  return acc != 0u;
}

constexpr int kPrepRows = 4;   // rows per warp and pass: their loads overlap

// One warp per group of kPrepRows rows: the row's largest |scaling * c| gives
// its exponent, then every value its digits, assembled in the warp's slice of
// shared memory and written with 16-byte stores.  A row's unit of 16 points
// is five 32-byte sectors, each the halves of points 0-7 and 8-15: the
// leading digits as FP16, then the biased bytes of digits 1, 2 | 3, 4 | 5, 6
// | 7 (the last one padded).  Bytes instead of FP16 planes: the tensor-core
// kernel gathers every row about 25 times, and the L2 gives all SMs together
// some 30 bytes per SM and clock - less than the tensor cores take of FP16
// planes (256 bytes a row and unit).
__global__ void __launch_bounds__(128) wide_prep_kernel(const __grid_constant__ WidePrep P) {
  extern __shared__ __align__(16) uint8_t s_stage[];
  grid_dep_launch();
  const DevDesc &d = P.d;
  const TreeDev &tr = P.tr;
  const int lane = threadIdx.x & 31;
  const int row_bytes = P.kp / kUnitK * kRowUnitBytes;
  uint8_t *stage = s_stage + (threadIdx.x >> 5) * kPrepRows * row_bytes;
  if (blockIdx.x == 0)
    for (int i = threadIdx.x; i < P.n_counters; i += blockDim.x) P.counters[i] = 0;
  if ((int)blockIdx.x >= P.row_blocks) {   // (uniform) the blocks that compare
    if (tree_differs(P, (blockIdx.x - P.row_blocks) * (int64_t)blockDim.x + threadIdx.x,
                     (int64_t)(gridDim.x - P.row_blocks) * blockDim.x)) {
      *P.stale = 1;
      reinterpret_cast<PlanStatus *>(P.st)->stale = 1;
    }
    return;
  }
  const int64_t n_rows = tr.nboxes * P.nv;
  const int64_t warps = (int64_t)P.row_blocks * (blockDim.x >> 5);
  const int cs = P.cc ? 2 : 1;
  for (int64_t grp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
       grp * kPrepRows < n_rows; grp += warps) {
    const int64_t r0 = grp * kPrepRows;
    const int n = (int)min((int64_t)kPrepRows, n_rows - r0);
    // lane j < n: row j's box data
    int cnt = 0, start = 0, level = 0, box = 0, v = 0;
    double sc = 0.0;
    if (lane < n) {
      box = (int)((r0 + lane) / P.nv);
      v = (int)((r0 + lane) - (int64_t)box * P.nv);
      cnt = tr.src_counts[box];
      if (cnt > d.nq) {
        report(P.st, VL1_E_LAYOUT, box, cnt);
        cnt = d.nq;
      }
      start = tr.src_starts[box];
      level = tr.levels[box];
      sc = box_scaling(d, tr, level);
    }
    int cnts[kPrepRows], sts[kPrepRows], exps[kPrepRows];
    double scs[kPrepRows];
    const double *c[kPrepRows];
    unsigned long long m[kPrepRows];
    int any = 0;
#pragma unroll
    for (int u = 0; u < kPrepRows; ++u) {
      cnts[u] = __shfl_sync(0xffffffffu, cnt, u);
      sts[u] = __shfl_sync(0xffffffffu, start, u);
      scs[u] = __shfl_sync(0xffffffffu, sc, u);
      const int vv = __shfl_sync(0xffffffffu, v, u);
      const int r = P.cc ? vv >> 1 : vv, part = P.cc ? vv & 1 : 0;
      if (u >= n) cnts[u] = 0;
      any = max(any, cnts[u]);
      c[u] = P.coefs + ((int64_t)r * tr.n_particles + sts[u]) * cs + part;
      m[u] = 0ull;
    }
    for (int k = lane; k < any; k += 32) {
      double x[kPrepRows];
#pragma unroll
      for (int u = 0; u < kPrepRows; ++u) x[u] = k < cnts[u] ? c[u][(int64_t)k * cs] : 0.0;
#pragma unroll
      for (int u = 0; u < kPrepRows; ++u) {
        const unsigned long long a =
            static_cast<unsigned long long>(__double_as_longlong(x[u])) & 0x7FFFFFFFFFFFFFFFull;
        m[u] = a > m[u] ? a : m[u];
      }
    }
#pragma unroll
    for (int u = 0; u < kPrepRows; ++u) {
      const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(m[u] >> 32));
      const unsigned lo = __reduce_max_sync(
          0xffffffffu, (unsigned)(m[u] >> 32) == hi ? (unsigned)m[u] : 0u);
      m[u] = ((unsigned long long)hi << 32) | lo;
      // rounding is monotone: the largest scaled value is that of the largest |c|
      const double top = scs[u] * __longlong_as_double((long long)m[u]);
      const unsigned long long tb = static_cast<unsigned long long>(__double_as_longlong(top)) &
                                    0x7FFFFFFFFFFFFFFFull;
      if (tb >= 0x7FF0000000000000ull) {
        exps[u] = kBadExp;
      } else if (tb == 0ull) {
        exps[u] = kZeroExp;
      } else {
        const int e = scale_exponent(top) - kTopBits;
        exps[u] = ((e + 8 * 4096 + 7) / 8) * 8 - 8 * 4096;   // up to a multiple of 8
      }
      if (lane == u && u < n) P.x_exp[r0 + u] = exps[u];
    }
    for (int k = lane * 16; k < kPrepRows * row_bytes; k += 32 * 16) {
      // zero digits: the first sector of a unit is FP16, the others are biased
      const unsigned z = k % kRowUnitBytes < 32 ? 0u : 0x80808080u;
      *reinterpret_cast<uint4 *>(stage + k) = make_uint4(z, z, z, z);
    }
    __syncwarp();
    for (int k = lane; k < any; k += 32) {
      double x[kPrepRows];
      int mode[kPrepRows];
#pragma unroll
      for (int u = 0; u < kPrepRows; ++u) {
        const bool have = k < cnts[u];
        x[u] = have ? c[u][(int64_t)k * cs] : 0.0;
        mode[u] = have ? tr.smode[sts[u] + k] : -2;
      }
#pragma unroll
      for (int u = 0; u < kPrepRows; ++u) {
        if (mode[u] == -2) continue;
        if (mode[u] < 0 || mode[u] >= d.nq) {
          report(P.st, VL1_E_LAYOUT, (int)((r0 + u) / P.nv), -1 - k);
          continue;
        }
        if (exps[u] == kBadExp || exps[u] == kZeroExp) continue;
        const double y = scs[u] * x[u];
        const RowDigits bd = row_digits(y, exps[u]);
        uint8_t *un = stage + u * row_bytes + (mode[u] / kUnitK) * kRowUnitBytes +
                      ((mode[u] >> 3) & 1) * 16;
        const int kk = mode[u] & 7;
        reinterpret_cast<__half *>(un)[kk] = __int2half_rn((int)(bd.hi >> 48));
#pragma unroll
        for (int i = 1; i < kW - 1; ++i)
          un[32 * ((i + 1) / 2) + 8 * ((i - 1) & 1) + kk] = (uint8_t)(bd.hi >> (8 * (6 - i)));
        un[32 * 4 + kk] = (uint8_t)bd.lo;
      }
    }
    __syncwarp();
    uint8_t *out = P.xpl + r0 * row_bytes;
    for (int k = lane * 16; k < n * row_bytes; k += 32 * 16)
      *reinterpret_cast<uint4 *>(out + k) = *reinterpret_cast<const uint4 *>(stage + k);
    if (P.wbox) {
      // 2D log displacement: sum_s c_s * dispfac(level) * nmlz[table level, s]
#pragma unroll
      for (int u = 0; u < kPrepRows; ++u) {
        if (u >= n) break;
        const int lvl = __shfl_sync(0xffffffffu, level, u);
        double re = 0.0, im = 0.0;
        if (cnts[u] > 0) {
          const double ext = level_extent(tr.root_extent, lvl);
          const double f = __dmul_rn(__dmul_rn(d.disp_coef, scs[u]),
                                     log(__ddiv_rn(ext, d.table_root_extent)));
          const int lev = pair_table_level(d, lvl);
          for (int k = lane; k < cnts[u]; k += 32) {
            const double x = c[u][(int64_t)k * cs];
            const int64_t ni = (int64_t)lev * d.nq + k;
            re = fma(x, f * (d.table_cplx ? d.nmlz[2 * ni] : d.nmlz[ni]), re);
            if (d.table_cplx) im = fma(x, f * d.nmlz[2 * ni + 1], im);
          }
        }
        for (int o = 16; o > 0; o >>= 1) {
          re += __shfl_xor_sync(0xffffffffu, re, o);
          if (d.table_cplx) im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (lane == 0) {
          P.wbox[2 * (r0 + u)] = re;
          P.wbox[2 * (r0 + u) + 1] = im;
        }
      }
    }
    __syncwarp();
  }
}

// ---------------------------------------------------------- main kernel

struct WideParams {
  DevDesc d;
  TreeDev tr;
  WideGeom g;
  int nv, cc;
  vl1_mixed_schedule sched;
  const uint8_t *xpl;
  const int *x_exp;
  const double *wbox;
  int n_xrows, n_keys;
  const __half *adig;
  const int *key_exp;      // per (table level, case) block
  longlong2 *partials;     // [slot][chunk][128][nch]: (S, L)
  int *counters;           // [split][chunk]
  const double *coefs;
  double *result;
  const int *stale;        // nonzero: the schedule is not this tree's (nullptr: it is)
  vl1_status *st;
  uint32_t wait_limit_us;
  int32_t withhold_arrival;
};

// Warp roles: 0-7 producers (16 tile rows each, two lanes per row), 8 table
// loader, 9 tensor-core issuer, 10.. readout (TMEM quadrant w % 4, 16 columns
// each).  One CTA per SM: at 64 output columns it has all 512 TMEM columns,
// and below that the registers of two CTAs would not do.
template <int NCH>
struct WideRoles {
  static constexpr int kProducers = 8;
  static constexpr int kLoader = kProducers;
  static constexpr int kMma = kProducers + 1;
  static constexpr int kRead0 = kProducers + 2;
  static constexpr int kRead = 4 * (NCH / 16);
  static constexpr int kThreads = 32 * (kRead0 + kRead);
  static constexpr int kStages = NCH >= 64 ? 4 : 5;   // 48 KB, 40 KB, 36 KB each
  static constexpr int kCtasPerSm = 1;
};
constexpr int kMaxStages = 5;
constexpr uint32_t kXPlaneBytes = 128u * kUnitK * 2u;

template <int NCH>
constexpr uint32_t wide_stage_bytes() {
  return kW * (kXPlaneBytes + (uint32_t)NCH * kUnitK * 2u);
}

struct WideBarriers {
  uint64_t xfull[kMaxStages], afull[kMaxStages], empty[kMaxStages];
  uint64_t fullA, fullB;     // accumulators d = 6 / d = 2..5 of a round complete
  uint64_t freeA, freeB;     // ... read out
  uint64_t drain;
};

// Products of a pipeline unit: density digit i times the stacked table digits
// j0 .. j0 + nb - 1, into the diagonals i + j0 ...  Part A covers d = 6..9,
// part B d = 2..5 (26 and 10 of the 36 digit pairs).  One set of accumulators
// (8 x NCH columns) has to do: a round's parts A and B of the first units
// (and of the last two) are issued A A A B B B, so that the readout of the
// previous round's d = 2..5 (complete with its last B: fullB, freeB) runs
// under three parts A and that of d = 6 (complete with its last A: fullA,
// freeA) under two parts B.  In plain A B A B order the issuer waited ~2,600
// of 10,000 clocks per round for the readout.
struct WideGroup {
  int i, j0, nb;
};
constexpr int kGroupsA = 8, kGroupsB = 4;
__device__ constexpr WideGroup kWideA[kGroupsA] = {{1, 5, 4}, {2, 4, 4}, {3, 3, 4}, {4, 2, 4},
                                                   {5, 1, 4}, {6, 1, 3}, {7, 1, 2}, {8, 1, 1}};
__device__ constexpr WideGroup kWideB[kGroupsB] = {{1, 1, 4}, {2, 1, 3}, {3, 1, 2}, {4, 1, 1}};

// two biased bytes of w (selector SEL of a byte permutation with 0x64) as
// FP16 digits: 0x64bb is 1024 + b, less 1152
template <unsigned SEL>
__device__ __forceinline__ uint32_t byte_digits(uint32_t w) {
  const uint32_t v = __byte_perm(w, 0x64646464u, SEL);
  const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&v), __float2half2_rn(1152.0f));
  return *reinterpret_cast<const uint32_t *>(&h);
}

// eight biased bytes as FP16 digits
__device__ __forceinline__ uint4 byte_row(uint32_t w0, uint32_t w1) {
  return make_uint4(byte_digits<0x4140>(w0), byte_digits<0x4342>(w0), byte_digits<0x4140>(w1),
                    byte_digits<0x4342>(w1));
}

template <int NCH>
__device__ __forceinline__ void wide_mma(uint32_t tbase, uint32_t x_lo, uint32_t a_lo, uint32_t hi,
                                         int i, int j0, int nb, uint32_t accumulate,
                                         uint32_t elected) {
  tc::mma_f16_elected(tbase + (uint32_t)(i + j0 - 2) * NCH,
                      x_lo + (((uint32_t)(i - 1) * kXPlaneBytes) >> 4),
                      a_lo + (((uint32_t)(j0 - 1) * NCH * kUnitK * 2u) >> 4), hi,
                      tc::idesc_f16_f32(128, NCH * nb), accumulate, elected);
}

// S 2^-48 + L 2^-72 (in units of 2^k) rounded once
__device__ __forceinline__ double wide_value(long long S, long long L, int k) {
  S += L >> 24;
  const long long rem = L & 0xFFFFFFll;
  if (S == 0 && rem == 0) return 0.0;
  const unsigned long long mag = S < 0 ? ~(unsigned long long)S : (unsigned long long)S;
  const int room = (mag ? __clzll((long long)mag) : 64) - 2;
  const int sh = room < 24 ? (room < 0 ? 0 : room) : 24;
  const long long tot = (long long)((unsigned long long)S << sh) + (rem >> (24 - sh));
  return scaled_i64_to_double(tot, k - 48 - sh);
}

// One target point of a row in FP64, the pairs in list order, from the tree's
// arrays alone: rows with non-finite sources, and all rows when the schedule is
// not the tree's.
__device__ __noinline__ void wide_slow_point(const WideParams &p, int tb, int r, int t) {
  const DevDesc &d = p.d;
  const TreeDev &tr = p.tr;
  const int tbox = tr.target_boxes[tb];
  const int tbeg = tr.tgt_starts[tbox];
  const int64_t ro = (int64_t)r * tr.n_particles;
  const bool oc = d.table_cplx || p.cc;
  const int tm = tr.tmode[tbeg + t];
  if (tm < 0 || tm >= d.nq) report(p.st, VL1_E_LAYOUT, tb, -1 - t);
  double a_re = 0.0, a_im = 0.0, w_re = 0.0, w_im = 0.0;
  for (int q = tr.starts[tb]; q < tr.starts[tb + 1] && tm >= 0 && tm < d.nq; ++q) {
    const int sbox = tr.lists[q];
    const int lvl = tr.levels[sbox];
    const double ext = level_extent(tr.root_extent, lvl);
    const int c = pair_case_id(d, tr, tbox, sbox, ext);
    if (c < 0) {
      if (t == 0) report(p.st, VL1_E_INVALID_CASE, tb, q);
      continue;
    }
    const int lev = pair_table_level(d, lvl);
    const double scl = pair_scaling(d, ext);
    const double df = d.disp_kind == VL1_DISP_LOG2D
                          ? __dmul_rn(__dmul_rn(d.disp_coef, scl),
                                      log(__ddiv_rn(ext, d.table_root_extent)))
                          : 0.0;
    const int sbeg = tr.src_starts[sbox], ns = min(tr.src_counts[sbox], d.nq);
    const int64_t blk = ((int64_t)lev * d.n_cases + c) * d.nq * d.nq;
    for (int s = 0; s < ns; ++s) {
      const int sm = tr.smode[sbeg + s];
      if (sm < 0 || sm >= d.nq) continue;
      const int64_t ci = ro + sbeg + s;
      const double c_re = p.cc ? p.coefs[2 * ci] : p.coefs[ci];
      const double c_im = p.cc ? p.coefs[2 * ci + 1] : 0.0;
      const int64_t bi = blk + (int64_t)sm * d.nq + tm;
      const double b_re = d.table_cplx ? d.blocks[2 * bi] : d.blocks[bi];
      const double x_re = c_re * scl, x_im = c_im * scl;
      a_re = fma(x_re, b_re, a_re);
      if (p.cc) a_im = fma(x_im, b_re, a_im);
      if (d.table_cplx) {
        const double b_im = d.blocks[2 * bi + 1];
        a_im = fma(x_re, b_im, a_im);
        if (p.cc) a_re = fma(-x_im, b_im, a_re);
      }
      if (d.disp_kind == VL1_DISP_LOG2D) {
        const int64_t ni = (int64_t)lev * d.nq + s;
        const double n_re = df * (d.table_cplx ? d.nmlz[2 * ni] : d.nmlz[ni]);
        const double n_im = d.table_cplx ? df * d.nmlz[2 * ni + 1] : 0.0;
        w_re += c_re * n_re - c_im * n_im;
        w_im += c_re * n_im + c_im * n_re;
      }
    }
  }
  const int64_t o = ro + tbeg + t;
  if (oc) {
    p.result[2 * o] = a_re + w_re;
    p.result[2 * o + 1] = a_im + w_im;
  } else {
    p.result[o] = a_re + w_re;
  }
}

template <int NCH>
__global__ void __launch_bounds__(WideRoles<NCH>::kThreads, WideRoles<NCH>::kCtasPerSm)
    wide_kernel(const __grid_constant__ WideParams p) {
  using R = WideRoles<NCH>;
  constexpr int kStages = R::kStages;
  constexpr uint32_t STAGE = wide_stage_bytes<NCH>();
  constexpr uint32_t COLS = 8 * NCH;
  constexpr int PARK = NCH + 1;   // padded rows: 32 lanes store one column conflict-free
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ WideBarriers bars;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int s_abort;
  __shared__ int s_row[128];       // tile row: j * nv + v, -1: empty
  __shared__ int s_E[128];         // the row's exponent: max of E + A over its sources
  __shared__ int s_bad[128];
  __shared__ int s_tbeg[128], s_cnt[128];   // the row's first target particle, its count
  __shared__ bool s_plain[128];             // its target points' modes are 0, 1, 2, ...
  __shared__ long long s_out[128];          // result index of that particle
  __shared__ double s_disp[128][2];
  __shared__ int s_any_bad, s_last, s_poison;
  __shared__ bool s_stale;
  __shared__ vl1_mixed_item s_item;   // kept here: the readout needs the registers

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t limit_us = p.wait_limit_us ? p.wait_limit_us : kWaitLimitUs;
  const bool withhold = p.withhold_arrival != 0 && blockIdx.x == 0 && blockIdx.y == 0;
  const int chunk = blockIdx.y;
  const int n_chunks = p.g.np / NCH;
  const int n_units_key = p.g.kp / kUnitK;

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) {
      tc::mbar_init(&bars.xfull[s], R::kProducers);   // one per producer warp
      tc::mbar_init(&bars.afull[s], 1);
      tc::mbar_init(&bars.empty[s], 1);
    }
    tc::mbar_init(&bars.fullA, 1);
    tc::mbar_init(&bars.fullB, 1);
    tc::mbar_init(&bars.freeA, R::kRead);
    tc::mbar_init(&bars.freeB, R::kRead);
    tc::mbar_init(&bars.drain, 1);
    tc::fence_mbar_init();
    s_abort = 0;
    s_any_bad = 0;
  }
  if (warp == R::kMma) {
    tc::tmem_alloc(&tmem_base, COLS);
    tc::tmem_relinquish();
  }

  if (tid == 0) {
    vl1_mixed_item item;
    if (p.sched.n_items > 0) {
      item = p.sched.items[blockIdx.x];
    } else {
      item.tile = blockIdx.x;
      item.key_begin = p.sched.tile_key_start[blockIdx.x];
      item.key_end = p.sched.tile_key_start[blockIdx.x + 1];
      item.split = -1;
      item.part = 0;
      item.nparts = 1;
      item.slot = -1;
    }
    bool ok = item.tile >= 0 && item.tile < p.sched.n_tiles && chunk < n_chunks;
    if (ok)
      ok = item.key_begin >= p.sched.tile_key_start[item.tile] &&
           item.key_end <= p.sched.tile_key_start[item.tile + 1] &&
           item.key_begin <= item.key_end;
    // (longer items' d = 7..9 sums could leave the int32 range unnoticed)
    const int n_keys = item.key_end - item.key_begin;
    ok = ok && (n_keys <= 1 || (int64_t)n_keys * p.g.kp <= kItemPoints);
    if (item.split >= 0)
      ok = ok && item.split < p.sched.n_splits && item.part >= 0 && item.part < item.nparts &&
           item.nparts < (1 << 16) && item.slot >= item.part &&
           item.slot - item.part + item.nparts <= p.sched.n_slots;
    if (!ok) {
      report(p.st, VL1_E_ARG, blockIdx.x, -1);
      item.split = -1;
      item.tile = -1;
      item.key_begin = item.key_end = 0;
    }
    s_item = item;
  }
  __syncthreads();

  if (tid < 128) {
    int v = s_item.tile >= 0 ? p.sched.tile_rows[(int64_t)s_item.tile * 128 + tid] : -1;
    if (v >= (int64_t)p.tr.n_tgt_boxes * p.nv) {
      report(p.st, VL1_E_ARG, s_item.tile, tid);
      v = -1;
    }
    int beg = 0, cnt = 0;
    long long o = 0;
    if (v >= 0) {
      const int j = v / p.nv, r = (v - j * p.nv) >> (p.cc ? 1 : 0);
      const int tbox = p.tr.target_boxes[j];
      beg = p.tr.tgt_starts[tbox];
      cnt = p.tr.tgt_counts[tbox];
      o = (long long)r * p.tr.n_particles + beg;
      if (cnt > p.d.nq) {
        report(p.st, VL1_E_LAYOUT, j, cnt);
        cnt = p.d.nq;
      }
    }
    s_tbeg[tid] = beg;
    s_cnt[tid] = cnt;
    s_out[tid] = o;
    s_row[tid] = v;
    s_E[tid] = kZeroExp;
    s_bad[tid] = 0;
  }
  grid_dep_wait();   // the density digits, their exponents and the split counters
  if (tid == 0) s_stale = p.stale && *reinterpret_cast<const volatile int *>(p.stale) != 0;
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tbase = tmem_base;

  // each row's exponent and displacement sum over its target box's list (all
  // of it: the parts of a split tile share them), which is the row's entries
  // of the tile's keys; kThreads / 128 threads per row
  {
    constexpr int NP = R::kThreads / 128;
    double *s_part = reinterpret_cast<double *>(smem);   // [NP][128][2]
    const int row = tid & 127, part = tid >> 7;
    if (part < NP) {
      int e = kZeroExp, bad = 0;
      double w_re = 0.0, w_im = 0.0;
      const bool have = s_row[row] >= 0;
      const int t0 = s_item.tile < 0 ? 0 : p.sched.tile_key_start[s_item.tile];
      const int t1 = s_item.tile < 0 ? 0 : p.sched.tile_key_start[s_item.tile + 1];
#pragma unroll 4
      for (int k = t0 + part; k < t1; k += NP) {
        const int xr = have ? p.sched.key_xrow[(int64_t)k * 128 + row] : -1;
        const int key = p.sched.key_ids[k];
        if (xr < 0 || xr >= p.n_xrows || key < 0 || key >= p.n_keys) continue;
        const int ex = p.x_exp[xr];
        if (ex == kBadExp)
          bad = 1;
        else
          e = max(e, ex + p.key_exp[key]);
        if (p.wbox) {
          w_re += p.wbox[2 * (int64_t)xr];
          w_im += p.wbox[2 * (int64_t)xr + 1];
        }
      }
      if (e > kZeroExp / 2) atomicMax(&s_E[row], e);
      if (bad) {
        s_bad[row] = 1;
        s_any_bad = 1;
      }
      if (p.wbox) {
        s_part[(part * 128 + row) * 2] = w_re;
        s_part[(part * 128 + row) * 2 + 1] = w_im;
      }
    }
    __syncthreads();
    if (p.wbox && tid < 128) {
      double re = 0.0, im = 0.0;
      for (int q = 0; q < NP; ++q) {
        re += s_part[(q * 128 + tid) * 2];
        im += s_part[(q * 128 + tid) * 2 + 1];
      }
      s_disp[tid][0] = re;
      s_disp[tid][1] = im;
    }
    if (p.wbox) __syncthreads();   // s_part lies in the stages
  }

  const int k0 = s_item.key_begin, k1 = s_stale ? k0 : s_item.key_end;
  const int n_units = (k1 - k0) * n_units_key;
  const int n_rounds = (n_units + kRoundUnits - 1) / kRoundUnits;

  if (warp < R::kProducers) {
    // ------------------------------------------------------------ producers
    // A lane holds one half (8 points) of one row: per unit it loads the
    // row's five 16-byte pieces two units ahead, turns the bytes into FP16 and
    // stores its 16 bytes of every plane into the stage's swizzled K-major
    // planes.  Source digit j goes to position j + shift, and the positions
    // below the shift are zero: (j + shift) % 8 takes digit j or zero.  The
    // planes lie a multiple of 128 bytes apart, so the lanes' banks do not
    // depend on the shift.
    const int my_row = 16 * warp + (lane >> 1), half = lane & 1;
    const int E = s_E[my_row];
    const uint32_t dst0 = tc::kmajor_swizzled_offset(my_row, half * 8, kUnitK);
    // the source row two keys ahead, and one key ahead its exponent too
    int key1 = -1, xr1 = -1, ex1 = kZeroExp, key2 = -1, xr2 = -1;
    auto fetch = [&](int k) {
      key2 = -1;
      xr2 = -1;
      if (k < k1) {
        key2 = p.sched.key_ids[k];
        xr2 = p.sched.key_xrow[(int64_t)k * 128 + my_row];
      }
    };
    auto advance = [&]() {
      key1 = key2;
      xr1 = xr2;
      ex1 = kZeroExp;
      if (xr1 >= p.n_xrows || key1 >= p.n_keys || (key1 < 0 && xr1 >= 0)) {
        report(p.st, VL1_E_ARG, s_item.tile, my_row);
        xr1 = -1;
      }
      if (xr1 >= 0) ex1 = p.x_exp[xr1] + p.key_exp[key1];
    };
    int kl = k0, kc = 0;               // the next unit to load
    const uint8_t *src = p.xpl;
    int shift = kW;
    struct Pieces {
      uint4 r[5];
      int shift;
    };
    auto load = [&](Pieces &b) {
      if (kc == 0) {
        // shift in digits; kW: the row is zero here (no source, or all digits
        // below the row's last one; rows with non-finite sources are summed
        // at the end)
        shift = kW;
        if (xr1 >= 0 && ex1 > kZeroExp / 2 && ex1 <= E) shift = min((E - ex1) >> 3, kW);
        src = p.xpl + ((int64_t)(xr1 < 0 ? 0 : xr1) * n_units_key) * kRowUnitBytes + half * 16;
        advance();
        fetch(kl + 2);
      }
      b.shift = shift;
      if (shift < kW) {
#pragma unroll
        for (int i = 0; i < 5; ++i)
          b.r[i] = __ldg(reinterpret_cast<const uint4 *>(src + kc * kRowUnitBytes + i * 32));
      }
      if (++kc == n_units_key) {
        kc = 0;
        ++kl;
      }
    };
    int s = 0;
    uint32_t ph = 1;                   // parity of the stage's previous release
    bool aborted = false;
    auto store = [&](const Pieces &b, int u) {
      if (u >= kStages && !wait_or_abort(&bars.empty[s], ph, &s_abort, limit_us, true)) {
        aborted = true;
        return;
      }
      uint8_t *xs = smem + (size_t)s * STAGE + dst0;
#pragma unroll
      for (int j = 0; j < kW; ++j) {
        // digit j: two words of piece (j + 1) / 2
        const uint4 q = b.r[(j + 1) / 2];
        uint4 v = j == 0 ? b.r[0] : ((j & 1) ? byte_row(q.x, q.y) : byte_row(q.z, q.w));
        if (j + b.shift >= kW) v = make_uint4(0u, 0u, 0u, 0u);
        *reinterpret_cast<uint4 *>(xs + (uint32_t)((j + b.shift) & (kW - 1)) * kXPlaneBytes) = v;
      }
      tc::fence_proxy_async_smem();    // generic writes before the tensor cores' reads
      __syncwarp();
      if (lane == 0 && !(withhold && warp == 0 && u == 0)) mbar_arrive(&bars.xfull[s]);
      if (++s == kStages) {
        s = 0;
        ph ^= 1u;
      }
    };
    fetch(k0);
    advance();
    fetch(k0 + 1);
    Pieces b0, b1;
    if (n_units > 0) load(b0);
    if (n_units > 1) load(b1);
    for (int u = 0; u < n_units; u += 2) {
      store(b0, u);
      if (aborted) break;
      if (u + 2 < n_units) load(b0);
      if (u + 1 >= n_units) break;
      store(b1, u + 1);
      if (aborted) break;
      if (u + 3 < n_units) load(b1);
    }
    __syncwarp();
  } else if (warp == R::kLoader) {
    // ---------------------------------------------------------- table loader
    if (lane == 0) {
      constexpr uint32_t ABYTES = kW * NCH * kUnitK * 2u;
      int u = 0;
      bool aborted = false;
      for (int kidx = k0; kidx < k1 && !aborted; ++kidx) {
        int key = p.sched.key_ids[kidx];
        if (key < 0 || key >= p.d.n_tables * p.d.n_cases) key = 0;   // reported by a producer
        for (int kc = 0; kc < n_units_key; ++kc, ++u) {
          const int s = u % kStages;
          const int use = u / kStages;
          if (use > 0 &&
              !wait_or_abort(&bars.empty[s], (use - 1) & 1, &s_abort, limit_us, false)) {
            aborted = true;
            break;
          }
          uint8_t *as = smem + (size_t)s * STAGE + kW * kXPlaneBytes;
          tc::mbar_arrive_expect_tx(&bars.afull[s], ABYTES);
          const int64_t tile = ((int64_t)key * n_units_key + kc) * n_chunks + chunk;
          tc::bulk_g2s(as, reinterpret_cast<const uint8_t *>(p.adig) + tile * ABYTES, ABYTES,
                       &bars.afull[s]);
        }
      }
      if (aborted || s_abort) {
        // copies of the last units may still be in flight into this CTA
        for (int v = u - kStages < 0 ? 0 : u - kStages; v < u; ++v)
          wait_bounded(&bars.afull[v % kStages], (v / kStages) & 1, limit_us);
      }
    }
    __syncwarp();
  } else if (warp == R::kMma) {
    // ------------------------------------------------------- tensor cores
    // The whole warp runs the loop (waits included) in step and one elected
    // lane executes the products, so that their operands are warp-uniform.
    const uint32_t el = tc::elect_one();
    const int total = __shfl_sync(0xffffffffu, n_units, 0);
    const uint32_t td = __shfl_sync(0xffffffffu, tbase, 0);
    const uint64_t desc0 = tc::smem_desc_kmajor_swizzled(tc::smem_addr(smem), kUnitK * 2);
    const uint32_t hi = (uint32_t)(desc0 >> 32);
    const uint32_t lo0 = __shfl_sync(0xffffffffu, (uint32_t)desc0, 0);
    auto wait = [&](uint64_t *bar, uint32_t phase) {
      return wait_or_abort(bar, phase, &s_abort, limit_us, false);
    };
    // The barriers of unit u + 1 are looked at between the products of unit u,
    // and waited for at its start only if they were not complete.
    bool aborted = false;
    int s = 0, in_round = 0;
    uint32_t ph = 0, round_ph = 1;     // parity of the previous round's release
    bool have_a = false, have_x = false, b_free = true, b_first = true;
    int pending = 0;                   // units whose part B is still to be issued
    for (int u = 0; u < total; ++u) {
      const bool first = in_round == 0;
      const int left = min(kRoundUnits, total - (u - in_round)) - 1 - in_round;   // in the round
      if ((!have_a && !wait(&bars.afull[s], ph)) || (!have_x && !wait(&bars.xfull[s], ph)) ||
          (first && u > 0 && !wait(&bars.freeA, round_ph))) {
        aborted = true;
        break;
      }
      tc::tc_fence_after();
      const uint32_t x_lo = lo0 + (((uint32_t)s * STAGE) >> 4);
      const uint32_t a_lo = x_lo + ((kW * kXPlaneBytes) >> 4);
      const int s_next = s + 1 == kStages ? 0 : s + 1;
      const uint32_t ph_next = s_next == 0 ? ph ^ 1u : ph;
      if (first) {
        b_free = u == 0;
        b_first = true;
        // d = 6 starts a round, d = 7..9 an item
        wide_mma<NCH>(td, x_lo, a_lo, hi, 1, 5, 1, 0u, el);
        wide_mma<NCH>(td, x_lo, a_lo, hi, 1, 6, 3, u == 0 ? 0u : 1u, el);
      } else {
        wide_mma<NCH>(td, x_lo, a_lo, hi, 1, 5, 4, 1u, el);
      }
      have_a = have_x = false;
#pragma unroll
      for (int g = 1; g < kGroupsA; ++g) {
        wide_mma<NCH>(td, x_lo, a_lo, hi, kWideA[g].i, kWideA[g].j0, kWideA[g].nb, 1u, el);
        if (u + 1 < total) {
          if (g == 2) have_a = tc::mbar_test(&bars.afull[s_next], ph_next);
          if (g == 4) have_x = tc::mbar_test(&bars.xfull[s_next], ph_next);
        }
      }
      if (left == 0) tc::mma_commit_elected(&bars.fullA, el);
      ++pending;
      // hold the first two units' parts B, and the last but one's, as long as
      // a stage stays free for the next unit
      const bool hold = left > 0 && (in_round < 2 || left == 1) && pending < kStages;
      if (!hold) {
        if (!b_free) {
          if (!wait(&bars.freeB, round_ph)) {
            aborted = true;
            break;
          }
          tc::tc_fence_after();
          b_free = true;
        }
        int sb = s - (pending - 1);
        if (sb < 0) sb += kStages;
        for (; pending > 0; --pending) {
          const uint32_t xb = lo0 + (((uint32_t)sb * STAGE) >> 4);
          const uint32_t ab = xb + ((kW * kXPlaneBytes) >> 4);
#pragma unroll
          for (int g = 0; g < kGroupsB; ++g)
            wide_mma<NCH>(td, xb, ab, hi, kWideB[g].i, kWideB[g].j0, kWideB[g].nb,
                          g == 0 && b_first ? 0u : 1u, el);
          b_first = false;
          tc::mma_commit_elected(&bars.empty[sb], el);   // stage free once these finish
          sb = sb + 1 == kStages ? 0 : sb + 1;
        }
        if (left == 0) tc::mma_commit_elected(&bars.fullB, el);
        if (u + 1 < total && !have_x) have_x = tc::mbar_test(&bars.xfull[s_next], ph_next);
      }
      s = s_next;
      ph = ph_next;
      if (left == 0) {
        in_round = 0;
        round_ph ^= 1u;
      } else {
        ++in_round;
      }
    }
    if (aborted || s_abort) {
      // products issued before the abort still write TMEM and read the stages
      tc::mma_commit_elected(&bars.drain, el);
      wait_bounded(&bars.drain, 0, limit_us);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ readout
    const int rw = warp - R::kRead0;
    const int quad = warp & 3;             // TMEM lanes 32 * quad .. + 31
    const int cb = rw >> 2;                // block of 16 columns
    const int row = quad * 32 + lane;
    const uint32_t col = tbase + ((uint32_t)(quad * 32) << 16) + cb * 16;
    // (the results' addressing, while the first round runs)
    for (int r = rw; r < 128; r += R::kRead) {
      bool same = true;
      for (int t = lane; t < s_cnt[r]; t += 32) same = same && p.tr.tmode[s_tbeg[r] + t] == t;
      same = __all_sync(0xffffffffu, same);
      if (lane == 0) s_plain[r] = same;
    }
    long long S[16];                       // d = 2..6, units 2^-48
#pragma unroll
    for (int c = 0; c < 16; ++c) S[c] = 0;
    bool ok = true;
    for (int round = 0; round < n_rounds; ++round) {
      if (!wait_or_abort(&bars.fullA, round & 1, &s_abort, limit_us, true)) {
        ok = false;
        break;
      }
      tc::tc_fence_after();
      uint32_t a[16];
      tc::tmem_ld16(col + 4 * NCH, a);     // d = 6
      tc::tmem_ld_wait();
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars.freeA);
#pragma unroll
      for (int c = 0; c < 16; ++c) S[c] += __float2int_rn(__uint_as_float(a[c]));
      if (!wait_or_abort(&bars.fullB, round & 1, &s_abort, limit_us, true)) {
        ok = false;
        break;
      }
      tc::tc_fence_after();
      // two diagonals of eight columns at a time (their loads together)
#pragma unroll
      for (int h = 0; h < 16; h += 8) {
        uint32_t b[8], c[8];
        tc::tmem_ld8(col + 3 * NCH + h, b);       // d = 5: weight 2^8
        tc::tmem_ld8(col + 2 * NCH + h, c);       // d = 4
        tc::tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i)
          S[h + i] += (long long)__float2int_rn(__uint_as_float(b[i])) * 256ll +
                      (long long)__float2int_rn(__uint_as_float(c[i])) * 65536ll;
        tc::tmem_ld8(col + NCH + h, b);           // d = 3
        tc::tmem_ld8(col + h, c);                 // d = 2: weight 2^32
        tc::tmem_ld_wait();
        if (h == 8) {
          tc::tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars.freeB);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
          S[h + i] +=
              (long long)__float2int_rn(__uint_as_float(b[i])) * 16777216ll +
              (long long)((unsigned long long)(unsigned)__float2int_rn(__uint_as_float(c[i]))
                          << 32);
      }
    }
    if (ok && !s_abort) {
      long long *s_S = reinterpret_cast<long long *>(smem);
      long long *s_L = s_S + 128 * PARK;
#pragma unroll
      for (int c = 0; c < 16; ++c) s_S[row * PARK + cb * 16 + c] = S[c];
      long long L[16];                     // d = 7..9, units 2^-72
#pragma unroll
      for (int c = 0; c < 16; ++c) L[c] = 0;
      if (n_rounds > 0) {
#pragma unroll 1
        for (int d = 7; d <= 9; ++d) {
          uint32_t a[16];
          tc::tmem_ld16(col + (d - 2) * NCH, a);
          tc::tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 16; ++c)
            L[c] = L[c] * 256ll + (long long)__float2int_rn(__uint_as_float(a[c]));
        }
      }
#pragma unroll
      for (int c = 0; c < 16; ++c) s_L[row * PARK + cb * 16 + c] = L[c];
    }
  }

  // ---- results: a split tile's parts store their exact sums, the part that
  // arrives last adds them in part order and writes
  tc::tc_fence_before();
  __syncthreads();
  long long *s_S = reinterpret_cast<long long *>(smem);
  long long *s_L = s_S + 128 * PARK;
  const vl1_mixed_item item = s_item;
  const bool stale = s_stale;
  bool write = !s_abort && item.tile >= 0 && !stale;
  if (item.split >= 0 && !stale) {
    // (a part that finds all others done keeps its sums in shared memory:
    // storing a part takes 17,000 clocks with every SM at it; 236 -> 233 us)
    int *const ctr = p.counters + (int64_t)item.split * n_chunks + chunk;
    if (tid == 0) s_last = (atomicAdd(ctr, 0) & 0xFFFF) == item.nparts - 1;
    __syncthreads();
    if (!s_abort && !s_last) {
      longlong2 *mine = p.partials + ((int64_t)item.slot * n_chunks + chunk) * 128 * NCH;
      for (int i = tid; i < 128 * NCH; i += R::kThreads) {
        const int o = (i / NCH) * PARK + i % NCH;
        mine[i] = make_longlong2(s_S[o], s_L[o]);
      }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      const int inc = s_abort ? (1 << 16) + 1 : 1;
      const int done = atomicAdd(ctr, inc) + inc;
      s_last = (done & 0xFFFF) == item.nparts;
      s_poison = done >> 16;
    }
    __syncthreads();
    write = write && s_last && !s_poison;
    if (write) {
      __threadfence();
      const longlong2 *all =
          p.partials + ((int64_t)(item.slot - item.part) * n_chunks + chunk) * 128 * NCH;
      const int64_t stride = (int64_t)n_chunks * 128 * NCH;
      constexpr int BATCH = 4;   // values per thread and pass, their loads together
      for (int i0 = tid; i0 < 128 * NCH; i0 += BATCH * R::kThreads) {
        long long S[BATCH] = {}, L[BATCH] = {};
        for (int q = 0; q < item.nparts; ++q) {
          if (q == item.part) continue;   // in shared memory
          longlong2 v[BATCH];
#pragma unroll
          for (int c = 0; c < BATCH; ++c) {
            const int i = i0 + c * R::kThreads;
            v[c] = i < 128 * NCH ? __ldcg(all + q * stride + i) : make_longlong2(0, 0);
          }
#pragma unroll
          for (int c = 0; c < BATCH; ++c) {
            S[c] += v[c].x;
            L[c] += v[c].y;
          }
        }
#pragma unroll
        for (int c = 0; c < BATCH; ++c) {
          const int i = i0 + c * R::kThreads;
          if (i < 128 * NCH) {
            s_S[(i / NCH) * PARK + i % NCH] += S[c];
            s_L[(i / NCH) * PARK + i % NCH] += L[c];
          }
        }
      }
    }
    __syncthreads();
  }
  if (write) {
    const bool tcx = p.d.table_cplx, pair = tcx && p.cc;
    const int cv = tcx ? 2 : 1;
    const int nq = p.d.nq;
    // A warp takes one output row at a time, lanes over the box's target
    // points, and four values per lane and pass (four rows, or two rows of
    // real and imaginary parts, or the four products of complex tables with
    // complex coefficients).
    constexpr int NW = R::kThreads / 32;
    const int n_out = pair ? 64 : 128, per = pair ? 1 : (tcx ? 2 : 4);
    for (int i0 = warp; i0 < n_out; i0 += per * NW) {
      for (int t = lane; t < nq; t += 32) {
        double y[4];
        bool on[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int i = i0 + (pair ? 0 : (tcx ? v >> 1 : v)) * NW;
          const int out = pair ? 2 * i : i;              // the output's row
          const int row = pair ? out + (v >> 1) : out;   // (odd rows: imaginary coefficients)
          on[v] = false;
          y[v] = 0.0;
          // rows with non-finite sources are summed below
          if (i >= n_out || t >= s_cnt[out] || s_bad[out] || (p.cc && s_bad[out ^ 1])) continue;
          const int m = s_plain[out] ? t : p.tr.tmode[s_tbeg[out] + t];
          const bool bad_mode = m < 0 || m >= nq;
          if (bad_mode && chunk == 0 && (!tcx || (pair ? v == 0 : (v & 1) == 0)))
            report(p.st, VL1_E_LAYOUT, s_row[out] / p.nv, -1 - t);
          const int col = (bad_mode ? 0 : m) * cv - chunk * NCH;
          if (col < 0 || col >= NCH) continue;
          on[v] = true;
          if (bad_mode) continue;
          const int part = tcx ? v & 1 : 0, at = row * PARK + col + part;
          y[v] = wide_value(s_S[at], s_L[at], s_E[row] + 2);
          if (p.wbox) y[v] += s_disp[row][part];
        }
        if (pair) {
          // (T_re + i T_im)(x_re + i x_im)
          if (on[0])
            reinterpret_cast<double2 *>(p.result)[s_out[2 * i0] + t] =
                make_double2(y[0] - y[3], y[1] + y[2]);
        } else if (tcx) {
#pragma unroll
          for (int j = 0; j < 2; ++j)
            if (on[2 * j])
              reinterpret_cast<double2 *>(p.result)[s_out[i0 + j * NW] + t] =
                  make_double2(y[2 * j], y[2 * j + 1]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (on[j]) {
              const long long o = s_out[i0 + j * NW] + t;
              if (p.cc)
                p.result[2 * o + (s_row[i0 + j * NW] & 1)] = y[j];
              else
                p.result[o] = y[j];
            }
        }
      }
    }
    if (s_any_bad) {
      __syncthreads();
      for (int row = 0; row < 128; ++row) {
        const int jv = s_row[row];
        if (jv < 0 || !s_bad[row]) continue;   // uniform
        const int j = jv / p.nv, v = jv - j * p.nv;
        // complex coefficients: both parts of an output once
        if (p.cc && (v & 1) && s_bad[row - 1]) continue;
        if (chunk == 0)
          for (int t = tid; t < s_cnt[row]; t += R::kThreads)
            wide_slow_point(p, j, p.cc ? v >> 1 : v, t);
      }
    }
  }
  if (stale && item.tile >= 0 && chunk == 0 && item.part == 0) {
    const int nq = p.d.nq;
    for (int i = tid; i < 128 * nq; i += R::kThreads) {
      const int row = i / nq, t = i - row * nq, jv = s_row[row];
      const int j = jv < 0 ? 0 : jv / p.nv, v = jv - j * p.nv;
      if (jv >= 0 && t < s_cnt[row] && !(p.cc && (v & 1)))
        wide_slow_point(p, j, p.cc ? v >> 1 : v, t);
    }
  }
  if (s_abort && tid == 0) report(p.st, VL1_E_TIMEOUT, item.tile, chunk);
  __syncthreads();
  if (warp == R::kMma) tc::tmem_dealloc(tbase, COLS);
}

template <int NCH>
size_t wide_smem() {
  const size_t pipe = (size_t)WideRoles<NCH>::kStages * wide_stage_bytes<NCH>();
  const size_t park = (size_t)2 * 128 * (NCH + 1) * 8;
  return (pipe > park ? pipe : park) + 1024;
}

template <int NCH>
cudaError_t launch_wide_kernel(const WideParams &p, dim3 grid, cudaStream_t s) {
  const size_t smem = wide_smem<NCH>();
  cudaError_t e = cudaFuncSetAttribute(wide_kernel<NCH>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  void *args[] = {const_cast<WideParams *>(&p)};
  return launch_overlapped(reinterpret_cast<const void *>(&wide_kernel<NCH>), grid,
                           dim3(WideRoles<NCH>::kThreads), args, smem, s);
}

int64_t round256(int64_t b) { return (b + 255) / 256 * 256; }

}  // namespace

WideGeom wide_geometry(int nq, int table_cplx) {
  WideGeom g;
  g.kp = ((nq + kUnitK - 1) / kUnitK) * kUnitK;
  const int n = table_cplx ? 2 * nq : nq;
  g.nch = n <= 16 ? 16 : (n <= 32 ? 32 : 64);
  g.np = ((n + g.nch - 1) / g.nch) * g.nch;
  return g;
}

int64_t wide_operand_bytes(const vl1_plan *plan) {
  const WideGeom g = wide_geometry(plan->d.nq, plan->d.table_cplx);
  const int64_t keys = (int64_t)plan->d.n_tables * plan->d.n_cases;
  return round256(keys * 4) + keys * g.kp * (int64_t)g.np * kW * 2;
}

// The plan's table digits, built on the first call that needs them (the
// stream is synchronised once, so that any stream can use them afterwards).
static int32_t wide_operands(vl1_plan *plan, cudaStream_t s) {
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  if (plan->wide.adig) return VL1_OK;
  const DevDesc &d = plan->d;
  const WideGeom g = wide_geometry(d.nq, d.table_cplx);
  const int64_t keys = (int64_t)d.n_tables * d.n_cases;
  const int64_t bytes = wide_operand_bytes(plan);
  if (plan->n_allocs >= (int)(sizeof(plan->allocs) / sizeof(plan->allocs[0]))) {
    set_error("internal: too many plan allocations");
    return VL1_E_NOMEM;
  }
  void *ptr = nullptr;
  cudaError_t e = lib_malloc_async(&ptr, (size_t)bytes, s);
  if (e != cudaSuccess) {
    set_error("stream-ordered allocation of %lld bytes failed: %s", (long long)bytes,
              cudaGetErrorString(e));
    cudaGetLastError();
    return VL1_E_NOMEM;
  }
  int *key_exp = static_cast<int *>(ptr);
  __half *adig = reinterpret_cast<__half *>(static_cast<uint8_t *>(ptr) +
                                            round256(keys * 4));
  wide_key_exp_kernel<<<(unsigned)keys, 256, 0, s>>>(d, plan->mixed.a_exp, key_exp);
  wide_digits_kernel<<<152 * 16, 256, 0, s>>>(d, g, key_exp, adig);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    cudaFreeAsync(ptr, s);
    return cuda_fail(e, "table digits of the FP64 tensor-core path");
  }
  plan->allocs[plan->n_allocs++] = ptr;
  plan->device_bytes += bytes;
  plan->wide.geom = g;
  plan->wide.key_exp = key_exp;
  plan->wide.adig = adig;
  return VL1_OK;
}

int32_t launch_wide(vl1_plan *plan, const TreeDev &tree, const vl1_tree_copy *made_from,
                    const vl1_mixed_schedule &sched, const double *coefs, int coef_cplx,
                    int nrhs, double *result, cudaStream_t s) {
  const DevDesc &d = plan->d;
  int32_t st = wide_operands(plan, s);
  if (st) return st;
  const WideGeom g = plan->wide.geom;
  const int nv = coef_cplx ? 2 * nrhs : nrhs;
  const int64_t n_rows = tree.nboxes * nv;
  const int n_chunks = g.np / g.nch;
  const bool disp = d.disp_kind == VL1_DISP_LOG2D;
  if (n_rows >= INT32_MAX || tree.nboxes < 1) {
    set_error("FP64 tensor-core path: %lld density rows exceed the 32-bit row index",
              (long long)n_rows);
    return VL1_E_UNSUPPORTED;
  }
  // scratch of this call, in stream order
  const int64_t b_exp = round256(n_rows * 4);
  const int64_t b_w = disp ? round256(n_rows * 16) : 0;
  const int64_t b_pl = round256(n_rows * (g.kp / kUnitK) * kRowUnitBytes);
  const int64_t b_ctr = round256((int64_t)sched.n_splits * n_chunks * 4 + 4);
  const int64_t b_part = (int64_t)sched.n_slots * n_chunks * 128 * g.nch * 16;
  void *scratch = nullptr;
  cudaError_t e =
      lib_malloc_async(&scratch, (size_t)(b_exp + b_w + b_pl + b_ctr + b_part), s);
  if (e != cudaSuccess) {
    set_error("scratch of the FP64 tensor-core path: %s", cudaGetErrorString(e));
    cudaGetLastError();
    return VL1_E_NOMEM;
  }
  uint8_t *w = static_cast<uint8_t *>(scratch);
  WidePrep pp;
  pp.d = d;
  pp.tr = tree;
  pp.coefs = coefs;
  pp.cc = coef_cplx;
  pp.nv = nv;
  pp.kp = g.kp;
  pp.x_exp = reinterpret_cast<int *>(w);
  w += b_exp;
  pp.wbox = disp ? reinterpret_cast<double *>(w) : nullptr;
  w += b_w;
  pp.xpl = w;
  w += b_pl;
  pp.counters = reinterpret_cast<int *>(w);
  w += b_ctr;
  pp.n_counters = sched.n_splits * n_chunks;
  pp.stale = made_from ? made_from->stale : nullptr;
  pp.max_chunks = 0;
  if (made_from) {
    const vl1_tree_view &c = made_from->tree;
    auto span = [&](int k, const void *now, const void *then, int64_t bytes) {
      const bool odd =
          ((reinterpret_cast<uintptr_t>(now) | reinterpret_cast<uintptr_t>(then)) & 15) != 0;
      pp.spans[k] = Span{static_cast<const uint8_t *>(now), static_cast<const uint8_t *>(then),
                         bytes, odd ? 0 : bytes / 16};
      if (pp.spans[k].chunks > pp.max_chunks) pp.max_chunks = pp.spans[k].chunks;
    };
    span(0, tree.smode, c.source_mode_ids, 4 * tree.n_particles);
    span(1, tree.lists, c.neighbor_source_boxes_lists, 4 * made_from->nnz);
    span(2, tree.starts, c.neighbor_source_boxes_starts, 4 * ((int64_t)tree.n_tgt_boxes + 1));
    span(3, tree.target_boxes, c.target_boxes, 4 * (int64_t)tree.n_tgt_boxes);
    span(4, tree.src_starts, c.box_source_starts, 4 * tree.nboxes);
    span(5, tree.src_counts, c.box_source_counts_nonchild, 4 * tree.nboxes);
    span(6, tree.levels, c.box_levels, tree.nboxes);
    span(7, tree.centers, c.box_centers, 8 * d.dim * tree.aligned_nboxes);
  }
  pp.st = plan->status;
  WideParams mp;
  mp.d = d;
  mp.tr = tree;
  mp.g = g;
  mp.nv = nv;
  mp.cc = coef_cplx;
  mp.sched = sched;
  mp.xpl = pp.xpl;
  mp.x_exp = pp.x_exp;
  mp.wbox = pp.wbox;
  mp.n_xrows = (int)n_rows;
  mp.n_keys = d.n_tables * d.n_cases;
  mp.adig = plan->wide.adig;
  mp.key_exp = plan->wide.key_exp;
  mp.partials = reinterpret_cast<longlong2 *>(w);
  mp.counters = pp.counters;
  mp.coefs = coefs;
  mp.result = result;
  mp.stale = made_from ? made_from->stale : nullptr;
  mp.st = plan->status;
  mp.wait_limit_us = g_test_wait_limit_us;
  mp.withhold_arrival = g_test_withhold;
  const size_t prep_smem = (size_t)4 * kPrepRows * (g.kp / kUnitK) * kRowUnitBytes;
  if (prep_smem > 48 * 1024)
    e = cudaFuncSetAttribute(wide_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)prep_smem);
  if (e == cudaSuccess) {
    const int64_t groups = (n_rows + kPrepRows - 1) / kPrepRows;
    // (blocks of their own compare the arrays, a thread one chunk of each: ahead
    // of the rows in the same blocks it took 4 us of 3D level 4, q = 5)
    pp.row_blocks = (int)std::min<int64_t>((groups + 3) / 4, 152 * 32);
    const int cmp =
        made_from ? (int)std::min<int64_t>(std::max<int64_t>((pp.max_chunks + 127) / 128, 1),
                                           152 * 16)
                  : 0;
    wide_prep_kernel<<<(unsigned)(pp.row_blocks + cmp), 128, prep_smem, s>>>(pp);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && sched.n_tiles > 0) {
    const dim3 grid(sched.n_items > 0 ? sched.n_items : sched.n_tiles, n_chunks);
    e = g.nch == 64 ? launch_wide_kernel<64>(mp, grid, s)
                    : (g.nch == 32 ? launch_wide_kernel<32>(mp, grid, s)
                                   : launch_wide_kernel<16>(mp, grid, s));
  }
  cudaFreeAsync(scratch, s);
  return e == cudaSuccess ? VL1_OK : cuda_fail(e, "FP64 tensor-core launch");
}

}  // namespace vl1
