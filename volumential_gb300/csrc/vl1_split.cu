// Helmholtz split correction: the list-1 point-to-point sum of the smooth
// remainder R = G_k - G_0 (Helmholtz minus Laplace), which the split mode
// adds to the Laplace-table near field
// (volumential/expansion_wrangler_fpnd.py:3491-3836, split order 1: the
// series remainder kernel of :212-332, strengths = density x quadrature
// weight, self pairs excluded by default).
//
//   2D: R(r) = c0 + sum_{n=1..N} (a_n log r + b_n) r^{2n}
//   3D: R(r) = sum_{n=1..N} c_n r^{n-1}
//
// with complex coefficients computed on the host.  FP64 throughout; a value of
// R costs ~2N FMAs and in 2D a logarithm, about 110 FP64 operations per point
// pair, on an FP64 pipe of two per SM and clock.
//
// The points of a box tree are one template per box, so R at a pair of points
// depends only on the pair of boxes' relative position and levels: on a tree
// of many boxes R is evaluated once per (source level, relative position) and
// point pair, and the sums read it from there (split_sum_kernel: two FMAs and
// 16 bytes per pair; bound by the FP64 pipe, 82 % busy, the tables in L1).
// split_mark_kernel checks on the device that every box's points are its
// level's template and every centre lies on the lattice (to a few ulps of the
// coordinates, the rounding of the points themselves) and its source and
// target points the same; otherwise, and for small trees, the per-pair kernel
// runs: one CTA per target box, one thread per target point, the points and
// strengths of each list-1 source box staged in shared memory.
//
// Measured (GB300, 2D k = 20, 102,400 points, 22.6M point pairs): 3,950 us per
// pair; with the tables 164 us on the device (sum 116, marking 30, tables 8,
// level boxes 6, the per-pair kernel that finds nothing to do 4).

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "vl1_internal.cuh"

namespace vl1 {
namespace {

constexpr int kSplitThreads = 128;
constexpr int kSplitMaxTerms = 128;

struct SplitArgs {
  int dim, n_points, nmax, exclude_self, wcplx, n_tgt_boxes;
  // 1: real wave number.  2D: the a_n are real and Im b_n = rho a_n, so two
  // real Horner sums give R; 3D: c_n is real for even n and imaginary for
  // odd n, so Re R and Im R are two Horner sums in r^2 over half the terms
  int real_k;
  double rho;
  const int32_t *target_boxes, *starts, *lists;
  const int32_t *src_starts, *src_counts, *tgt_starts, *tgt_counts;
  const double *points;    // [dim][n_points]
  const double *weights;   // [n_points] or [n_points][2]
  const double *coef;      // [2][nmax + 1][2]: (a_n | c_n) then (b_n), (re, im); index 0: c0
  double *result;          // [n_points][2]
};

// R at squared distance r2 from the coefficients in shared memory
template <int DIM>
__device__ __forceinline__ void remainder_value(const SplitArgs &A,
                                                const double (*s_coef)[kSplitMaxTerms + 1][2],
                                                double r2, double &re, double &im) {
  if (DIM == 2 && A.real_k) {
    double pa = s_coef[0][A.nmax][0], pb = s_coef[1][A.nmax][0];
    for (int n = A.nmax - 1; n >= 1; --n) {
      pa = fma(pa, r2, s_coef[0][n][0]);
      pb = fma(pb, r2, s_coef[1][n][0]);
    }
    const double lg = r2 > 0.0 ? 0.5 * log(r2) : 0.0;
    re = s_coef[0][0][0] + r2 * fma(lg, pa, pb);
    im = fma(A.rho * r2, pa, s_coef[0][0][1]);
  } else if (DIM == 3 && A.real_k) {
    const double r = sqrt(r2);
    // Re R = r sum_{m>=1} c_{2m} r2^(m-1), Im R = sum_{m>=0} Im c_{2m+1} r2^m
    const int me = A.nmax / 2, mo = (A.nmax - 1) / 2;
    double pe = me >= 1 ? s_coef[0][2 * me][0] : 0.0;
    for (int m = me - 1; m >= 1; --m) pe = fma(pe, r2, s_coef[0][2 * m][0]);
    double po = s_coef[0][2 * mo + 1][1];
    for (int m = mo - 1; m >= 0; --m) po = fma(po, r2, s_coef[0][2 * m + 1][1]);
    re = r * pe;
    im = po;
  } else if (DIM == 2) {
    // Horner in x = r^2 for the log and power series (terms n >= 1)
    double pa_re = s_coef[0][A.nmax][0], pa_im = s_coef[0][A.nmax][1];
    double pb_re = s_coef[1][A.nmax][0], pb_im = s_coef[1][A.nmax][1];
    for (int n = A.nmax - 1; n >= 1; --n) {
      pa_re = fma(pa_re, r2, s_coef[0][n][0]);
      pa_im = fma(pa_im, r2, s_coef[0][n][1]);
      pb_re = fma(pb_re, r2, s_coef[1][n][0]);
      pb_im = fma(pb_im, r2, s_coef[1][n][1]);
    }
    // the log term is dropped at r = 0 (its factor r^{2n} vanishes;
    // any nonzero r2 in FP64 has r far above 1e-300)
    const double lg = r2 > 0.0 ? 0.5 * log(r2) : 0.0;
    re = s_coef[0][0][0] + r2 * fma(lg, pa_re, pb_re);
    im = s_coef[0][0][1] + r2 * fma(lg, pa_im, pb_im);
  } else {
    const double r = sqrt(r2);
    re = s_coef[0][A.nmax][0];
    im = s_coef[0][A.nmax][1];
    for (int n = A.nmax - 1; n >= 1; --n) {
      re = fma(re, r, s_coef[0][n][0]);
      im = fma(im, r, s_coef[0][n][1]);
    }
  }
}

__device__ __forceinline__ void load_coefficients(const SplitArgs &A,
                                                  double (*s_coef)[kSplitMaxTerms + 1][2]) {
  for (int i = threadIdx.x; i < 2 * (A.nmax + 1); i += blockDim.x) {
    const int part = i / (A.nmax + 1), n = i - part * (A.nmax + 1);
    s_coef[part][n][0] = A.coef[(part * (A.nmax + 1) + n) * 2];
    s_coef[part][n][1] = A.coef[(part * (A.nmax + 1) + n) * 2 + 1];
  }
  __syncthreads();
}

// Tables of R by relative position (see the top of the file).
constexpr int kSplitLevels = 32;
constexpr int kSplitBase = 13;           // offsets -6 .. 6 quarters of the source box
struct SplitTables {
  int nq, max_slots, n_codes;
  int64_t aligned_nboxes, nboxes;
  double root_extent;
  const double *centers;                 // [dim][aligned_nboxes]
  const uint8_t *levels;
  int *bad;          // nonzero: the per-pair kernel runs
  int *n_slots;
  int *level_box;    // [kSplitLevels]: a box of the level with points, or -1
  int *slot_of;      // [kSplitLevels][3][n_codes]: table of (source level, level step, offset)
  int2 *slot_key;    // [max_slots]: (source level * 3 + step + 1, code)
  double2 *table;    // [max_slots][nq (source)][nq (target)]
};

// the key of a pair of boxes, or -1: source level, target level - source level
// (-1, 0, 1) and centre offset in quarters of the source box.  CHECK false: a
// pair that split_mark_kernel has accepted.
template <int DIM, bool CHECK>
__device__ __forceinline__ int split_key(const SplitTables &T, int tb, int sb) {
  const int ls = T.levels[sb], step = (int)T.levels[tb] - ls;
  if (CHECK && (ls >= kSplitLevels || step < -1 || step > 1)) return -1;
  const double quarter = 0.25 * T.root_extent / (double)(1ll << ls);
  int code = 0;
#pragma unroll
  for (int a = 0; a < DIM; ++a) {
    const double ct = T.centers[a * T.aligned_nboxes + tb];
    const double cs = T.centers[a * T.aligned_nboxes + sb];
    const double r = rint((ct - cs) / quarter);
    code = code * kSplitBase + (int)r + 6;
    if (!CHECK) continue;
    // the boxes of one tree lie on its lattice, up to the centres' rounding
    // (a centre is the root vertex plus a part of the root extent): the same
    // few ulps that the points are held to, since the tables take the lattice
    // position for the distance
    const double ulp = 2.220446049250313e-16 * (fabs(ct) + fabs(cs) + T.root_extent);
    if (!(fabs((ct - cs) - r * quarter) <= 2.0 * ulp) || fabs(r) > 6.0) return -1;
  }
  return (ls * 3 + step + 1) * T.n_codes + code;
}

// a box of every level that has points (any: they are compared with it)
__global__ void split_level_kernel(const SplitArgs A, const SplitTables T) {
  for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < T.nboxes;
       b += (int64_t)gridDim.x * blockDim.x) {
    if (A.src_counts[b] <= 0) continue;
    if (T.levels[b] >= kSplitLevels)
      *T.bad = 1;
    else
      atomicMax(T.level_box + T.levels[b], (int)b);
  }
}

// Checks that a box's points are its level's template around its centre and
// gives every (source level, position) of list 1 a table.  One warp per box /
// target box.
template <int DIM>
__global__ void split_mark_kernel(const SplitArgs A, const SplitTables T) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t b = warp; b < T.nboxes; b += warps) {
    const int cnt = A.src_counts[b];
    if (cnt <= 0 && A.tgt_counts[b] <= 0) continue;
    const int ref = T.levels[b] < kSplitLevels ? T.level_box[T.levels[b]] : -1;
    bool ok = cnt == T.nq && A.tgt_counts[b] == cnt && A.src_starts[b] == A.tgt_starts[b] &&
              ref >= 0 && A.src_counts[ref] == cnt;
    for (int i = lane; ok && i < cnt; i += 32)
#pragma unroll
      for (int a = 0; a < DIM; ++a) {
        const double cb = T.centers[a * T.aligned_nboxes + b];
        const double cr = T.centers[a * T.aligned_nboxes + ref];
        const double xb = A.points[(int64_t)a * A.n_points + A.src_starts[b] + i];
        const double xr = A.points[(int64_t)a * A.n_points + A.src_starts[ref] + i];
        const double ulp = 2.220446049250313e-16 * (fabs(xb) + fabs(xr) + fabs(cb) + fabs(cr));
        ok = ok && fabs((xb - cb) - (xr - cr)) <= 2.0 * ulp;
      }
    if (!__all_sync(0xffffffffu, ok) && lane == 0) *T.bad = 1;
  }
  for (int64_t i = warp; i < A.n_tgt_boxes; i += warps)
    for (int q = A.starts[i] + lane; q < A.starts[i + 1]; q += 32) {
      // (boxes without points need no table, and their levels may have none)
      if (A.tgt_counts[A.target_boxes[i]] <= 0 || A.src_counts[A.lists[q]] <= 0) continue;
      const int key = split_key<DIM, true>(T, A.target_boxes[i], A.lists[q]);
      // (two boxes in one place: the table of the position has no self pairs)
      constexpr int kHere = DIM == 2 ? 6 * kSplitBase + 6 : (6 * kSplitBase + 6) * kSplitBase + 6;
      const bool twin = key >= 0 && A.lists[q] != A.target_boxes[i] &&
                        (key / T.n_codes) % 3 == 1 && key % T.n_codes == kHere;
      if (key < 0 || twin) {
        *T.bad = 1;
      } else if (T.slot_of[key] < 0 && atomicCAS(T.slot_of + key, -1, -2) == -1) {
        const int slot = atomicAdd(T.n_slots, 1);
        if (slot < T.max_slots) {
          T.slot_key[slot] = make_int2(key / T.n_codes, key % T.n_codes);
          T.slot_of[key] = slot;
        } else {
          *T.bad = 1;
        }
      }
    }
}

// R of every table entry; the excluded self pairs are zero
template <int DIM>
__global__ void __launch_bounds__(kSplitThreads)
    split_table_kernel(const SplitArgs A, const SplitTables T) {
  __shared__ double s_coef[2][kSplitMaxTerms + 1][2];
  if (*T.bad) return;
  load_coefficients(A, s_coef);
  const int64_t per = (int64_t)T.nq * T.nq, n = (int64_t)*T.n_slots * per;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int slot = (int)(i / per), st = (int)(i - slot * per);
    const int s = st / T.nq, t = st - s * T.nq;
    const int2 key = T.slot_key[slot];
    const int ls = key.x / 3, lt = ls + key.x % 3 - 1;
    const int bs = T.level_box[ls], bt = T.level_box[lt];
    const double quarter = 0.25 * T.root_extent / (double)(1ll << ls);
    double r2 = 0.0;
    int code = key.y;
    bool same = ls == lt && s == t;
#pragma unroll
    for (int a = DIM - 1; a >= 0; --a) {
      const int off = code % kSplitBase - 6;
      code /= kSplitBase;
      same = same && off == 0;
      const double xs = A.points[(int64_t)a * A.n_points + A.src_starts[bs] + s] -
                        T.centers[a * T.aligned_nboxes + bs];
      const double xt = A.points[(int64_t)a * A.n_points + A.src_starts[bt] + t] -
                        T.centers[a * T.aligned_nboxes + bt];
      const double d = (double)off * quarter + (xt - xs);
      r2 = fma(d, d, r2);
    }
    double re = 0.0, im = 0.0;
    if (!(same && A.exclude_self)) remainder_value<DIM>(A, s_coef, r2, re, im);
    T.table[i] = make_double2(re, im);
  }
}

// The sums: one CTA per target box, a thread one target point and every
// `split`-th source point; consecutive threads read consecutive targets.
constexpr int kSplitChunk = 9;   // source boxes staged together
template <int DIM>
__global__ void __launch_bounds__(256)
    split_sum_kernel(const SplitArgs A, const SplitTables T, int split) {
  extern __shared__ __align__(16) double s_dyn[];   // strengths, then the split's sums
  if (*T.bad) return;
  const int nq = T.nq;
  double2 *s_w = reinterpret_cast<double2 *>(s_dyn), *s_red = s_w + kSplitChunk * nq;
  const int tb = A.target_boxes[blockIdx.x];
  if (A.tgt_counts[tb] <= 0) return;
  const int t = threadIdx.x % nq, sg = threadIdx.x / nq;
  __shared__ int s_slot[kSplitChunk], s_src[kSplitChunk];
  __shared__ bool s_self[kSplitChunk];
  double re = 0.0, im = 0.0;
  const int q_end = A.starts[blockIdx.x + 1];
  for (int q0 = A.starts[blockIdx.x]; q0 < q_end; q0 += kSplitChunk) {
    const int m = min(kSplitChunk, q_end - q0);
    __syncthreads();
    if (threadIdx.x < m) {   // one thread per source box: its table and points
      const int sb = A.lists[q0 + threadIdx.x];
      const bool have = A.src_counts[sb] > 0;
      s_slot[threadIdx.x] = have ? T.slot_of[split_key<DIM, false>(T, tb, sb)] : -1;
      s_src[threadIdx.x] = A.src_starts[sb];
      s_self[threadIdx.x] = A.exclude_self && sb == tb;
    }
    __syncthreads();
    // strengths of the chunk's sources
    for (int i = threadIdx.x; i < m * nq; i += blockDim.x) {
      const int p = i / nq;
      const int64_t s = s_src[p] + (i - p * nq);
      if (s_slot[p] >= 0)
        s_w[i] = A.wcplx ? make_double2(A.weights[2 * s], A.weights[2 * s + 1])
                         : make_double2(A.weights[s], 0.0);
    }
    __syncthreads();
    if (sg >= split) continue;
    for (int p = 0; p < m; ++p) {
      if (s_slot[p] < 0) continue;
      const double2 *R = T.table + (int64_t)s_slot[p] * nq * nq + t;
      const double2 *w = s_w + p * nq;
      // an excluded self pair adds nothing, whatever its weight (the table's
      // zero times an infinite or NaN weight would be NaN)
      const int skip = s_self[p] ? t : -1;
      if (A.wcplx) {
#pragma unroll 4
        for (int s = sg; s < nq; s += split) {
          const double2 r = __ldg(R + (int64_t)s * nq);
          const double2 v = s == skip ? make_double2(0.0, 0.0) : w[s];
          re = fma(v.x, r.x, fma(-v.y, r.y, re));
          im = fma(v.x, r.y, fma(v.y, r.x, im));
        }
      } else {
#pragma unroll 8
        for (int s = sg; s < nq; s += split) {
          const double2 r = __ldg(R + (int64_t)s * nq);
          const double v = s == skip ? 0.0 : w[s].x;
          re = fma(v, r.x, re);
          im = fma(v, r.y, im);
        }
      }
    }
  }
  __syncthreads();
  if (sg < split) s_red[sg * nq + t] = make_double2(re, im);
  __syncthreads();
  if (sg == 0) {
    for (int g = 1; g < split; ++g) {
      re += s_red[g * nq + t].x;
      im += s_red[g * nq + t].y;
    }
    const int64_t o = A.tgt_starts[tb] + t;
    A.result[2 * o] = re;
    A.result[2 * o + 1] = im;
  }
}

template <int DIM>
__global__ void __launch_bounds__(kSplitThreads) split_remainder_kernel(const SplitArgs A,
                                                                       const int *only_if) {
  __shared__ double s_pts[DIM][kSplitThreads];
  __shared__ double s_w[2][kSplitThreads];
  __shared__ int s_idx[kSplitThreads];
  __shared__ double s_coef[2][kSplitMaxTerms + 1][2];
  if (only_if && !*only_if) return;   // the tables serve this tree
  load_coefficients(A, s_coef);
  const int tb = A.target_boxes[blockIdx.x];
  const int t0 = A.tgt_starts[tb], nt = A.tgt_counts[tb];
  for (int tbase = 0; tbase < nt; tbase += kSplitThreads) {
    const int ti = tbase + threadIdx.x;
    const bool have_t = ti < nt;
    const int tgt = have_t ? t0 + ti : 0;
    double x[DIM];
#pragma unroll
    for (int a = 0; a < DIM; ++a) x[a] = have_t ? A.points[(int64_t)a * A.n_points + tgt] : 0.0;
    double acc_re = 0.0, acc_im = 0.0;
    for (int p = A.starts[blockIdx.x]; p < A.starts[blockIdx.x + 1]; ++p) {
      const int sb = A.lists[p];
      const int s0 = A.src_starts[sb], ns = A.src_counts[sb];
      for (int sbase = 0; sbase < ns; sbase += kSplitThreads) {
        const int m = min(kSplitThreads, ns - sbase);
        __syncthreads();
        if (threadIdx.x < m) {
          const int s = s0 + sbase + threadIdx.x;
#pragma unroll
          for (int a = 0; a < DIM; ++a) s_pts[a][threadIdx.x] = A.points[(int64_t)a * A.n_points + s];
          s_w[0][threadIdx.x] = A.wcplx ? A.weights[2 * (int64_t)s] : A.weights[s];
          s_w[1][threadIdx.x] = A.wcplx ? A.weights[2 * (int64_t)s + 1] : 0.0;
          s_idx[threadIdx.x] = s;
        }
        __syncthreads();
        if (!have_t) continue;
        for (int j = 0; j < m; ++j) {
          if (A.exclude_self && s_idx[j] == tgt) continue;
          double r2 = 0.0;
#pragma unroll
          for (int a = 0; a < DIM; ++a) {
            const double d = x[a] - s_pts[a][j];
            r2 = fma(d, d, r2);
          }
          double re, im;
          remainder_value<DIM>(A, s_coef, r2, re, im);
          const double wr = s_w[0][j], wi = s_w[1][j];
          acc_re = fma(wr, re, fma(-wi, im, acc_re));
          acc_im = fma(wr, im, fma(wi, re, acc_im));
        }
      }
    }
    if (have_t) {
      A.result[2 * (int64_t)tgt] = acc_re;
      A.result[2 * (int64_t)tgt + 1] = acc_im;
    }
  }
}

// Target boxes from which the tables are tried: with ~9 (2D) or ~20 (3D)
// source boxes each, at most 33 (139) positions per level pair and a few
// levels, R is then evaluated for a small part of the pairs; the extra
// launches cost about 20 us.
constexpr int kSplitTableBoxes = 512;
constexpr int64_t kSplitTableBytes = 128ll << 20;

template <int DIM>
int32_t launch_split(const SplitArgs &A, const vl1_tree_view &V, cudaStream_t s) {
  int *only_if = nullptr;
  void *scratch = nullptr;
  cudaError_t e = cudaSuccess;
  const int n_boxes = (int)V.nboxes;
  // a box's point count, if the tree is uniform in it: n_points per target
  // box (checked on the device)
  const int nq = A.n_points / A.n_tgt_boxes;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  e = cudaStreamIsCapturing(s, &cap);
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamIsCapturing");
  if (A.n_tgt_boxes >= kSplitTableBoxes && nq >= 2 && nq <= 256 &&
      (int64_t)nq * A.n_tgt_boxes == A.n_points && V.box_centers && V.box_levels && n_boxes > 0 &&
      V.root_extent > 0.0 && cap == cudaStreamCaptureStatusNone) {
    SplitTables T;
    T.nq = nq;
    T.n_codes = DIM == 2 ? kSplitBase * kSplitBase : kSplitBase * kSplitBase * kSplitBase;
    T.aligned_nboxes = V.aligned_nboxes;
    T.nboxes = V.nboxes;
    T.root_extent = V.root_extent;
    T.centers = V.box_centers;
    T.levels = V.box_levels;
    const int64_t per = (int64_t)nq * nq * 16;
    T.max_slots = (int)std::min<int64_t>(kSplitTableBytes / per, 4096);
    const int64_t n_keys = (int64_t)kSplitLevels * 3 * T.n_codes;
    const int64_t head = 2 + kSplitLevels + n_keys;    // bad, n_slots, level_box, slot_of
    const int64_t head_bytes = (head * 4 + 255) / 256 * 256;
    const int64_t key_bytes = ((int64_t)T.max_slots * 8 + 255) / 256 * 256;
    e = lib_malloc_async(&scratch, (size_t)(head_bytes + key_bytes + T.max_slots * per), s);
    if (e == cudaSuccess) {
      uint8_t *w = static_cast<uint8_t *>(scratch);
      T.bad = reinterpret_cast<int *>(w);
      T.n_slots = T.bad + 1;
      T.level_box = T.bad + 2;
      T.slot_of = T.level_box + kSplitLevels;
      T.slot_key = reinterpret_cast<int2 *>(w + head_bytes);
      T.table = reinterpret_cast<double2 *>(w + head_bytes + key_bytes);
      only_if = T.bad;
      e = cudaMemsetAsync(T.bad, 0, 8, s);
      if (e == cudaSuccess) e = cudaMemsetAsync(T.level_box, 0xFF, 4 * (head - 2), s);
      if (e == cudaSuccess) {
        split_level_kernel<<<std::min((n_boxes + 255) / 256, 1024), 256, 0, s>>>(A, T);
        split_mark_kernel<DIM><<<std::min((n_boxes + 7) / 8, 152 * 8), 256, 0, s>>>(A, T);
        split_table_kernel<DIM><<<152 * 8, kSplitThreads, 0, s>>>(A, T);
        const int split = std::max(1, std::min(8, (nq <= 128 ? 192 : 256) / nq));
        const int threads = (nq * split + 31) / 32 * 32;
        const size_t smem = 16 * (size_t)nq * (kSplitChunk + split);
        split_sum_kernel<DIM><<<A.n_tgt_boxes, threads, smem, s>>>(A, T, split);
        e = cudaGetLastError();
      }
      if (e != cudaSuccess) {
        cudaFreeAsync(scratch, s);
        return cuda_fail(e, "split table launch");
      }
    } else {
      cudaGetLastError();   // no scratch: the per-pair kernel
      scratch = nullptr;
    }
  }
  split_remainder_kernel<DIM><<<A.n_tgt_boxes, kSplitThreads, 0, s>>>(A, only_if);
  e = cudaGetLastError();
  if (scratch) cudaFreeAsync(scratch, s);
  return e == cudaSuccess ? VL1_OK : cuda_fail(e, "split_remainder_kernel launch");
}

}  // namespace
}  // namespace vl1

using namespace vl1;

extern "C" int32_t vl1_split_correction(const vl1_split_desc *desc, void *stream) {
  if (!desc || !desc->tree || !desc->points || !desc->weights || !desc->coefficients ||
      !desc->result) {
    set_error("vl1_split_correction: null argument");
    return VL1_E_ARG;
  }
  const vl1_split_desc &D = *desc;
  const vl1_tree_view &T = *D.tree;
  if ((D.dim != 2 && D.dim != 3) || D.n_points < 0 || D.n_terms < 1 ||
      D.n_terms > kSplitMaxTerms || T.n_target_boxes < 0) {
    set_error("vl1_split_correction: dim %d, %d points or %d series terms out of range",
              D.dim, D.n_points, D.n_terms);
    return VL1_E_ARG;
  }
  if (T.n_target_boxes == 0) return VL1_OK;
  if (!T.target_boxes || !T.neighbor_source_boxes_starts || !T.neighbor_source_boxes_lists ||
      !T.box_source_starts || !T.box_source_counts_nonchild || !T.box_target_starts ||
      !T.box_target_counts_nonchild) {
    set_error("vl1_split_correction: null array in the tree view");
    return VL1_E_ARG;
  }
  SplitArgs A;
  A.dim = D.dim;
  A.n_points = D.n_points;
  A.nmax = D.n_terms;
  A.exclude_self = D.exclude_self;
  A.wcplx = D.weights_complex;
  A.n_tgt_boxes = T.n_target_boxes;
  A.real_k = (D.flags & VL1_SPLIT_REAL_K) ? 1 : 0;
  A.rho = -0.5 * 3.14159265358979323846;   // Im b_n / a_n for a real wave number
  A.target_boxes = T.target_boxes;
  A.starts = T.neighbor_source_boxes_starts;
  A.lists = T.neighbor_source_boxes_lists;
  A.src_starts = T.box_source_starts;
  A.src_counts = T.box_source_counts_nonchild;
  A.tgt_starts = T.box_target_starts;
  A.tgt_counts = T.box_target_counts_nonchild;
  A.points = D.points;
  A.weights = D.weights;
  A.coef = D.coefficients;
  A.result = D.result;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  return D.dim == 2 ? launch_split<2>(A, T, s) : launch_split<3>(A, T, s);
}
