// FP64 table builder: singular box integrals by the Duffy radial scheme.
//
// Each table entry (case, source mode, target point) is
//   T = int_{[0,h]^d} G(t - y) phi_m(y) dy
// with t the case's target point, phi_m the source mode's tensor Lagrange
// basis on the Gauss-Legendre nodes of [0, h], and G a free-space kernel.
// The scheme of the reference's batched builder
// (volumential/nearfield_potential_table.py:2035-2223 for the integrand,
// :2225-2291 for the nodes): the box is split at the target point clipped
// into it into 2^d sub-boxes (one per sign vector; empty ones dropped), each
// sub-box into d! simplices (one per axis order), and each simplex is
// mapped from the unit cube by the Duffy map u_{perm(i)} = prod_{k<=i} r_k,
// whose Jacobian prod_{i<d-1} r_i^(d-1-i) cancels the singularity at the
// target; r_0 (radial) takes a tanh-sinh rule, r_1.. a Gauss-Legendre rule.
//
// The node count per target is 2^d d! n_reg^(d-1) n_rad (3D, default orders:
// 8 x 6 x 400 x 123 = 2.4M) and the FP64 pipe bounds both kernels below.
//
// duffy_group_kernel (radial kernels): all q^d modes of one target together.
// On a simplex the coordinate along the i-th axis of its order is
// dc + s r_0 .. r_i, so the sums over r_{d-1}, .., r_0 nest: for a fixed
// (r_0, .., r_{d-2}) the last axis' basis functions are polynomials of
// degree q - 1 in r_{d-1}, and the sum over r_{d-1} is taken once against
// the Lagrange basis on q Chebyshev points xi_k of [0, 1] (moments M_k, one
// FMA per k and node), then turned into all q modes through their values at
// r_0 .. r_{d-2} xi_k.  Per node: the distance, one kernel value and q FMAs,
// against the kernel value and d (q - 1) products per node *and entry* of
// duffy_entry_kernel.  Every FP64 operation of a node counts: the kernel's
// constant factor and the basis' weights multiply the sums instead, and the
// test for a zero distance is an integer one (3D Laplace q = 4: 12.3 -> 10.8
// ms a build).
//
// Measured (GB300, default orders, whole build calls): 3D Laplace q = 4
// (12,936 entries, 636 targets) 370 -> 10.5 ms, 3D Helmholtz q = 4 604 -> 30 ms,
// 2D Helmholtz q = 5 4.4 -> 1.4 ms; entries within 1e-15 of the per-entry
// sums, relative to the largest.
//
// duffy_entry_kernel (plane waves, derivatives, q beyond the instances): one
// CTA per entry and simplex, threads striding over the nodes.

#include <cuda_runtime.h>

#include <cstdint>

#include <algorithm>

#include "vl1_internal.cuh"

namespace vl1 {
namespace {

constexpr int kDuffyThreads = 256;
constexpr int kDuffyMaxQ = 16;

struct DuffyArgs {
  vl1_duffy_desc d;
  int n_perm, n_reg_tail, n_sub, n_chunks;
  double *part;   // [entry][chunk][re, im] partial sums
};

// axis orders in itertools.permutations order
__device__ constexpr int8_t kPerm2[2][2] = {{0, 1}, {1, 0}};
__device__ constexpr int8_t kPerm3[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2},
                                            {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};

// d/dt_a of G(dvec) (dvec = target - source) times the scaling constant,
// Laplace and Helmholtz: G'(r) d_a / r; (re, im)
template <int DIM>
__device__ __forceinline__ void green_gradient(int kind, double k, int axis, const double *dv,
                                               double &re, double &im) {
  double r2 = 0.0;
#pragma unroll
  for (int a = 0; a < DIM; ++a) r2 = fma(dv[a], dv[a], r2);
  const double da = dv[axis];
  im = 0.0;
  switch (kind) {
    case VL1_DUFFY_LAPLACE2D:   // -d_a / (2 pi r^2)
      re = -da / r2 * (0.5 / 3.141592653589793);
      break;
    case VL1_DUFFY_LAPLACE3D:   // -d_a / (4 pi r^3)
      re = -da / (r2 * sqrt(r2)) * (0.25 / 3.141592653589793);
      break;
    case VL1_DUFFY_HELMHOLTZ2D: {   // -(i/4) k H1(k r) d_a / r = (k/4)(Y1 - i J1) d_a / r
      const double r = sqrt(r2);
      const double f = 0.25 * k * da / r;
      re = f * y1(k * r);
      im = -f * j1(k * r);
      break;
    }
    default: {   // VL1_DUFFY_HELMHOLTZ3D: exp(i k r) (i k r - 1) d_a / (4 pi r^3)
      const double r = sqrt(r2);
      double sn, cs;
      sincos(k * r, &sn, &cs);
      const double f = (0.25 / 3.141592653589793) * da / (r2 * r);
      // (cs + i sn)(-1 + i k r) = (-cs - k r sn) + i (k r cs - sn)
      re = f * (-cs - k * r * sn);
      im = f * (k * r * cs - sn);
      break;
    }
  }
}

// G(dvec) times the kernel's scaling constant; (re, im)
template <int DIM>
__device__ __forceinline__ void green(int kind, double k, int power, const double *dv,
                                      double &re, double &im) {
  double r2 = 0.0;
#pragma unroll
  for (int a = 0; a < DIM; ++a) r2 = fma(dv[a], dv[a], r2);
  im = 0.0;
  switch (kind) {
    case VL1_DUFFY_LAPLACE2D:   // -log(r) / (2 pi)
      re = -0.5 * log(r2) * (0.5 / 3.141592653589793);
      break;
    case VL1_DUFFY_LAPLACE3D:   // 1 / (4 pi r)
      re = rsqrt(r2) * (0.25 / 3.141592653589793);
      break;
    case VL1_DUFFY_HELMHOLTZ2D: {   // (i/4) H0^(1)(k r) = (-Y0 + i J0) / 4
      const double kr = k * sqrt(r2);
      re = -0.25 * y0(kr);
      im = 0.25 * j0(kr);
      break;
    }
    case VL1_DUFFY_HELMHOLTZ3D: {   // exp(i k r) / (4 pi r)
      const double r = sqrt(r2);
      double s, c;
      sincos(k * r, &s, &c);
      const double f = (0.25 / 3.141592653589793) / r;
      re = c * f;
      im = s * f;
      break;
    }
    case VL1_DUFFY_CONSTANT:
      re = 1.0;
      break;
    case VL1_DUFFY_POWER:
    case VL1_DUFFY_POWER_LOG: {   // r^p (times log r): r2^(p/2), times r for odd p
      double v = 1.0;
      for (int i = 0; i < power / 2; ++i) v *= r2;
      if (power & 1) v *= sqrt(r2);
      re = kind == VL1_DUFFY_POWER ? v : v * (0.5 * log(r2));
      break;
    }
    default:   // VL1_DUFFY_PLANE_WAVE: cos(k d_0)
      re = cos(k * dv[0]);
      break;
  }
}

// One CTA per (entry, chunk) work item, or a capped grid striding over them:
// a chunk is one (sign vector, axis order) of the entry's Duffy
// sub-simplices, so an item runs for a fraction of a millisecond; the partial
// sums are added per entry in chunk order by duffy_reduce_kernel (a fixed
// order: the table is the same on every run, whatever the grid).
template <int DIM>
__global__ void __launch_bounds__(kDuffyThreads) duffy_entry_kernel(const DuffyArgs A) {
  const vl1_duffy_desc &D = A.d;
  constexpr int dim = DIM;
  const int q = D.q;
  __shared__ double s_xi[kDuffyMaxQ], s_bw[kDuffyMaxQ];
  __shared__ double s_red[2][kDuffyThreads / 32];
  if (threadIdx.x < q) {
    s_xi[threadIdx.x] = D.interp_nodes[threadIdx.x];
    s_bw[threadIdx.x] = D.interp_weights[threadIdx.x];
  }
  __syncthreads();
  // work item w = (entry, chunk); a capped grid strides over them
  const int n_chunks = A.n_chunks;
  const int64_t n_work = (int64_t)D.n_entries * n_chunks;
  for (int64_t item = blockIdx.x; item < n_work; item += gridDim.x) {
  const int e = (int)(item / n_chunks);
  const int chunk = (int)(item - (int64_t)e * n_chunks);   // isub * n_perm + iperm
  double t[3], dc[3];
  int mode[3];
  bool mode_ok = true;
#pragma unroll
  for (int a = 0; a < dim; ++a) {
    t[a] = D.target_points[(int64_t)a * D.n_entries + e];
    dc[a] = D.decomposition_targets[(int64_t)a * D.n_entries + e];
    mode[a] = D.mode_axes[(int64_t)a * D.n_entries + e];
    mode_ok = mode_ok && mode[a] >= 0 && mode[a] < q;
  }
  double *part = A.part + ((int64_t)e * n_chunks + chunk) * 2;
  if (!mode_ok) {   // an invalid entry yields NaN (the host checks its inputs)
    if (threadIdx.x == 0) {
      part[0] = __longlong_as_double(0x7FF8000000000000ll);
      part[1] = __longlong_as_double(0x7FF8000000000000ll);
    }
    continue;   // uniform across the CTA
  }
  const int iperm = chunk % A.n_perm;
  const int isub = chunk / A.n_perm;
  const int64_t n_nodes = (int64_t)A.n_reg_tail * D.n_rad;   // nodes of this chunk
  double acc_re = 0.0, acc_im = 0.0;
  for (int64_t i = threadIdx.x; i < n_nodes; i += kDuffyThreads) {
    // node index -> (regular tail node, radial node)
    const int irad = (int)(i % D.n_rad);
    int ireg = (int)(i / D.n_rad);
    // sub-box lengths along each axis (sign bit of axis a: first axis slowest)
    double len[3], sg[3];
    bool active = true;
    double len_prod = 1.0;
#pragma unroll
    for (int a = 0; a < dim; ++a) {
      sg[a] = ((isub >> (dim - 1 - a)) & 1) ? 1.0 : -1.0;
      len[a] = sg[a] < 0.0 ? dc[a] : D.extent - dc[a];
      active = active && len[a] > 0.0;
      len_prod *= len[a];
    }
    if (!active) continue;
    // unit-cube coordinates r_0 (radial), r_1.. (regular; first slowest)
    double rs[3];
    rs[0] = D.radial_nodes[irad];
    double w = D.radial_weights[irad];
#pragma unroll
    for (int a = dim - 1; a >= 1; --a) {
      const int j = ireg % D.n_reg;
      ireg /= D.n_reg;
      rs[a] = D.regular_nodes[j];
      w *= D.regular_weights[j];
    }
    // Duffy map and its Jacobian
    double cumv[3], cum = 1.0;
#pragma unroll
    for (int i2 = 0; i2 < dim; ++i2) {
      cum *= rs[i2];
      cumv[i2] = cum;
    }
    // u[perm[i2]] = cumv[i2], written as u[a] = cumv[position of a in perm]
    double u[3];
#pragma unroll
    for (int a = 0; a < dim; ++a) {
      double v = 0.0;
#pragma unroll
      for (int i2 = 0; i2 < dim; ++i2) {
        const int axis = dim == 3 ? kPerm3[iperm][i2] : kPerm2[iperm][i2];
        v = axis == a ? cumv[i2] : v;
      }
      u[a] = v;
    }
    double jac = 1.0;
#pragma unroll
    for (int i2 = 0; i2 < dim - 1; ++i2)
#pragma unroll
      for (int p = 0; p < dim - 1 - i2; ++p) jac *= rs[i2];
    // source point, displacement (target - source) and the mode's basis
    double dv[3], basis = 1.0;
#pragma unroll
    for (int a = 0; a < dim; ++a) {
      const double y = fma(sg[a] * len[a], u[a], dc[a]);
      dv[a] = t[a] - y;
      if (q > 1) {
        // first-form Lagrange polynomial: bw_m prod_{j != m} (y - x_j)
        double l = s_bw[mode[a]];
        for (int j = 0; j < q; ++j)
          if (j != mode[a]) l *= y - s_xi[j];
        basis *= l;
      }
    }
    double r2 = 0.0;
#pragma unroll
    for (int a = 0; a < dim; ++a) r2 = fma(dv[a], dv[a], r2);
    if (!(r2 > 0.0)) continue;   // a node on the singular point: zero weight
    double gre, gim;
    if (D.derivative == 0) {
      green<DIM>(D.kernel, D.k, D.power, dv, gre, gim);
    } else {
      const int axis = (D.derivative > 0 ? D.derivative : -D.derivative) - 1;
      green_gradient<DIM>(D.kernel, D.k, axis, dv, gre, gim);
      if (D.derivative < 0) {   // d/dy_a G(t - y) = -d/dt_a G
        gre = -gre;
        gim = -gim;
      }
    }
    const double f = w * jac * len_prod * basis;
    acc_re = fma(gre, f, acc_re);
    acc_im = fma(gim, f, acc_im);
  }
  // CTA reduction
  for (int o = 16; o > 0; o >>= 1) {
    acc_re += __shfl_down_sync(0xffffffffu, acc_re, o);
    acc_im += __shfl_down_sync(0xffffffffu, acc_im, o);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    s_red[0][warp] = acc_re;
    s_red[1][warp] = acc_im;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double re = 0.0, im = 0.0;
    for (int w2 = 0; w2 < kDuffyThreads / 32; ++w2) {
      re += s_red[0][w2];
      im += s_red[1][w2];
    }
    part[0] = re;
    part[1] = im;
  }
  __syncthreads();   // s_red is reused by the next work item
  }
}

// the entries' values: their chunks' partial sums added in chunk order
__global__ void duffy_reduce_kernel(const double *part, int n_entries, int n_chunks,
                                    int complex_output, double *out) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n_entries;
       e += gridDim.x * blockDim.x) {
    double re = 0.0, im = 0.0;
    for (int c = 0; c < n_chunks; ++c) {
      re += part[((int64_t)e * n_chunks + c) * 2];
      im += part[((int64_t)e * n_chunks + c) * 2 + 1];
    }
    if (complex_output) {
      out[2 * (int64_t)e] = re;
      out[2 * (int64_t)e + 1] = im;
    } else {
      out[e] = re;
    }
  }
}

// ---------------------------------------------- all modes of a target

// G(r) for the radial kernels, up to the factor green_factor(kind), which the
// group kernel applies once per sum instead of once per node
__host__ __device__ constexpr double green_factor(int kind) {
  return kind == VL1_DUFFY_LAPLACE2D ? -0.25 / 3.141592653589793
         : kind == VL1_DUFFY_LAPLACE3D || kind == VL1_DUFFY_HELMHOLTZ3D
             ? 0.25 / 3.141592653589793
             : 1.0;
}
__device__ __forceinline__ void green_radial(int kind, double k, int power, double r2,
                                             double &re, double &im) {
  im = 0.0;
  switch (kind) {
    case VL1_DUFFY_LAPLACE2D:   // -log(r) / (2 pi) = -log(r^2) / (4 pi)
      re = log(r2);
      break;
    case VL1_DUFFY_LAPLACE3D:   // 1 / (4 pi r)
      re = rsqrt(r2);
      break;
    case VL1_DUFFY_HELMHOLTZ2D: {
      const double kr = k * sqrt(r2);
      re = -0.25 * y0(kr);
      im = 0.25 * j0(kr);
      break;
    }
    case VL1_DUFFY_HELMHOLTZ3D: {   // exp(i k r) / (4 pi r)
      const double r = sqrt(r2);
      double s, c;
      sincos(k * r, &s, &c);
      const double f = 1.0 / r;
      re = c * f;
      im = s * f;
      break;
    }
    case VL1_DUFFY_CONSTANT:
      re = 1.0;
      break;
    default: {   // VL1_DUFFY_POWER, VL1_DUFFY_POWER_LOG
      double v = 1.0;
      for (int i = 0; i < power / 2; ++i) v *= r2;
      if (power & 1) v *= sqrt(r2);
      re = kind == VL1_DUFFY_POWER ? v : v * (0.5 * log(r2));
      break;
    }
  }
}

// The Q Lagrange polynomials on the nodes x at y without their weights (the
// products of the differences to the other nodes, from the left and from the
// right; the weights are applied once per sum).
template <int Q>
__device__ __forceinline__ void node_products(double y, const double *x, double (&l)[Q]) {
  double d[Q];
#pragma unroll
  for (int m = 0; m < Q; ++m) d[m] = y - x[m];
  double left = 1.0;
#pragma unroll
  for (int m = 0; m < Q; ++m) {
    l[m] = left;
    left = m == 0 ? d[0] : left * d[m];
  }
  double right = 1.0;
#pragma unroll
  for (int m = Q - 1; m >= 0; --m) {
    l[m] = m == Q - 1 ? l[m] : (m == 0 ? right : l[m] * right);
    right = m == Q - 1 ? d[m] : right * d[m];
  }
}

struct DuffyGroupArgs {
  vl1_duffy_desc d;
  int n_groups, n_perm, n_chunks;
  const int32_t *group_entry;   // an entry with the group's target
  double *part;                 // [group][chunk][mode][re (, im)]
};

constexpr int kGroupThreads = 128;
// radial nodes below this carry no weight that a double could hold beside
// the others (their products with the Jacobian are below 1e-60), and their
// distances could leave the FP64 range
constexpr double kLeastRadius = 1e-60;

template <int DIM, int Q, bool CPLX>
constexpr int group_smem_doubles(int n_reg) {
  constexpr int NU = (DIM == 3 ? Q * Q : Q) * (CPLX ? 2 : 1);
  return 3 * Q + n_reg * (2 + Q) + kGroupThreads * (NU + 1 + Q);
}

// One CTA per (target, simplex) work item, or a capped grid striding over
// them; a thread takes one radial node at a time and sums over the regular
// nodes, its sums over the last d - 1 axes' modes in registers (U), and the
// CTA then contracts them with the first axis' basis over its radial nodes.
template <int DIM, int Q, bool CPLX>
__global__ void __launch_bounds__(kGroupThreads) duffy_group_kernel(const DuffyGroupArgs A) {
  const vl1_duffy_desc &D = A.d;
  constexpr int CV = CPLX ? 2 : 1;
  constexpr int NU = (DIM == 3 ? Q * Q : Q) * CV;
  constexpr int NM = (DIM == 3 ? Q * Q * Q : Q * Q) * CV;   // outputs
  constexpr int US = NU + 1;   // odd strides: the contraction reads a column of a thread each
  extern __shared__ __align__(16) double sm[];
  double *s_x = sm, *s_bw = s_x + Q, *s_xi = s_bw + Q;
  double *s_r = s_xi + Q, *s_w = s_r + D.n_reg, *s_phi = s_w + D.n_reg;   // [n_reg][Q]
  double *s_u = s_phi + D.n_reg * Q, *s_l0 = s_u + kGroupThreads * US;    // [thread][..]
  const int tid = threadIdx.x;
  if (tid < Q) {
    s_x[tid] = D.interp_nodes[tid];
    s_bw[tid] = D.interp_weights[tid];
    s_xi[tid] = 0.5 - 0.5 * cospi((2 * tid + 1) / (2.0 * Q));
  }
  __syncthreads();
  for (int i = tid; i < D.n_reg; i += kGroupThreads) {
    s_r[i] = D.regular_nodes[i];
    s_w[i] = D.regular_weights[i];
    for (int k = 0; k < Q; ++k) {   // weight x Lagrange basis on the Chebyshev points
      double v = D.regular_weights[i];
      for (int j = 0; j < Q; ++j)
        if (j != k) v *= (D.regular_nodes[i] - s_xi[j]) / (s_xi[k] - s_xi[j]);
      s_phi[i * Q + k] = v;
    }
  }
  __syncthreads();
  const int64_t n_work = (int64_t)A.n_groups * A.n_chunks;
  for (int64_t item = blockIdx.x; item < n_work; item += gridDim.x) {
    const int g = (int)(item / A.n_chunks), chunk = (int)(item - (int64_t)g * A.n_chunks);
    const int e = A.group_entry[g];
    const int iperm = chunk % A.n_perm, isub = chunk / A.n_perm;
    double *part = A.part + item * NM;
    // along axis a: source coordinate dc + s c, displacement b - s c
    double dc[3] = {}, b[3] = {}, s[3] = {};
    bool active = true;
    double len_prod = 1.0;
#pragma unroll
    for (int i = 0; i < DIM; ++i) {   // in the order of the simplex
      const int a = DIM == 3 ? kPerm3[iperm][i] : kPerm2[iperm][i];
      const double t = D.target_points[(int64_t)a * D.n_entries + e];
      dc[i] = D.decomposition_targets[(int64_t)a * D.n_entries + e];
      b[i] = t - dc[i];
      const bool up = (isub >> (DIM - 1 - a)) & 1;
      const double len = up ? D.extent - dc[i] : dc[i];
      active = active && len > 0.0;
      len_prod *= len;
      s[i] = up ? len : -len;
    }
    if (!active) {   // uniform: an empty sub-box
      for (int m = tid; m < NM; m += kGroupThreads) part[m] = 0.0;
      continue;
    }
    double sum[(NM + kGroupThreads - 1) / kGroupThreads] = {};
    for (int i0 = 0; i0 < D.n_rad; i0 += kGroupThreads) {
      const int i = i0 + tid;
      const double r0 = i < D.n_rad ? D.radial_nodes[i] : 0.0;
      double u[NU];
#pragma unroll
      for (int n = 0; n < NU; ++n) u[n] = 0.0;
      if (r0 >= kLeastRadius) {
        const double d0 = fma(-s[0], r0, b[0]);
        const double base0 = d0 * d0;
        const int n1 = DIM == 3 ? D.n_reg : 1;
        for (int j1 = 0; j1 < n1; ++j1) {
          const double a = DIM == 3 ? r0 * s_r[j1] : r0;
          double base = base0;
          if (DIM == 3) {
            const double d1 = fma(-s[1], a, b[1]);
            base = fma(d1, d1, base0);
          }
          const double c = s[DIM - 1] * a;
          double mom[Q * CV];
#pragma unroll
          for (int k = 0; k < Q * CV; ++k) mom[k] = 0.0;
#pragma unroll 2
          for (int j2 = 0; j2 < D.n_reg; ++j2) {
            const double d2 = fma(-c, s_r[j2], b[DIM - 1]);
            const double r2 = fma(d2, d2, base);
            double gre = 0.0, gim = 0.0;
            // r2 > 0 (a sum of squares), tested off the FP64 pipe
            if ((unsigned long long)(__double_as_longlong(r2) - 1ll) < 0x7FF0000000000000ull)
              green_radial(D.kernel, D.k, D.power, r2, gre, gim);
#pragma unroll
            for (int k = 0; k < Q; ++k) {
              mom[k * CV] = fma(gre, s_phi[j2 * Q + k], mom[k * CV]);
              if (CPLX) mom[k * CV + 1] = fma(gim, s_phi[j2 * Q + k], mom[k * CV + 1]);
            }
          }
          // the last axis' modes from the moments
          double tm[Q * CV];
#pragma unroll
          for (int k = 0; k < Q * CV; ++k) tm[k] = 0.0;
#pragma unroll
          for (int k = 0; k < Q; ++k) {
            double l[Q];
            node_products<Q>(fma(c, s_xi[k], dc[DIM - 1]), s_x, l);
#pragma unroll
            for (int m = 0; m < Q; ++m) {
              tm[m * CV] = fma(l[m], mom[k * CV], tm[m * CV]);
              if (CPLX) tm[m * CV + 1] = fma(l[m], mom[k * CV + 1], tm[m * CV + 1]);
            }
          }
          if (DIM == 3) {
            double l[Q];
            node_products<Q>(fma(s[1], a, dc[1]), s_x, l);
            const double w1 = s_w[j1] * s_r[j1];
#pragma unroll
            for (int m1 = 0; m1 < Q; ++m1) {
              const double lw = l[m1] * w1;
#pragma unroll
              for (int m = 0; m < Q * CV; ++m)
                u[m1 * Q * CV + m] = fma(lw, tm[m], u[m1 * Q * CV + m]);
            }
          } else {
#pragma unroll
            for (int m = 0; m < Q * CV; ++m) u[m] = tm[m];
          }
        }
      }
      double l[Q];
      node_products<Q>(fma(s[0], r0, dc[0]), s_x, l);
      const double w0 = i < D.n_rad ? D.radial_weights[i] * len_prod *
                                          (DIM == 3 ? r0 * r0 : r0)
                                    : 0.0;
#pragma unroll
      for (int m = 0; m < Q; ++m) s_l0[tid * Q + m] = l[m] * w0;
#pragma unroll
      for (int n = 0; n < NU; ++n) s_u[tid * US + n] = u[n];
      __syncthreads();
      const int n_act = min(kGroupThreads, D.n_rad - i0);
#pragma unroll
      for (int o = 0; o < (NM + kGroupThreads - 1) / kGroupThreads; ++o) {
        const int m = o * kGroupThreads + tid;
        if (m < NM) {
          const int m0 = m / NU, n = m - m0 * NU;
          double v = sum[o];
          for (int q = 0; q < n_act; ++q) v = fma(s_l0[q * Q + m0], s_u[q * US + n], v);
          sum[o] = v;
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int o = 0; o < (NM + kGroupThreads - 1) / kGroupThreads; ++o) {
      const int m = o * kGroupThreads + tid;
      if (m < NM) {
        // simplex order (m0, m1, (m2)) to axis order, axis 0 slowest
        int rest = m / CV, mode = 0;
        double factor = green_factor(D.kernel);
#pragma unroll
        for (int i = DIM - 1; i >= 0; --i) {
          const int a = DIM == 3 ? kPerm3[iperm][i] : kPerm2[iperm][i];
          int stride = 1;
          for (int x = a; x < DIM - 1; ++x) stride *= Q;
          mode += (rest % Q) * stride;
          factor *= s_bw[rest % Q];
          rest /= Q;
        }
        part[mode * CV + m % CV] = sum[o] * factor;
      }
    }
  }
}

// the entries' values: the partial sums of their target and mode over the
// simplices, in order (a fixed one, whatever the grid)
__global__ void duffy_group_reduce_kernel(const vl1_duffy_desc D, const double *part,
                                          const int32_t *entry_group, int n_chunks, int cv,
                                          double *out) {
  const int nm = (D.dim == 3 ? D.q * D.q * D.q : D.q * D.q) * cv;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < D.n_entries;
       e += gridDim.x * blockDim.x) {
    int mode = 0;
    bool ok = true;
    for (int a = 0; a < D.dim; ++a) {
      const int m = D.mode_axes[(int64_t)a * D.n_entries + e];
      ok = ok && m >= 0 && m < D.q;
      mode = mode * D.q + m;
    }
    double re = 0.0, im = 0.0;
    if (ok) {
      const double *p = part + (int64_t)entry_group[e] * n_chunks * nm + mode * cv;
      for (int c = 0; c < n_chunks; ++c) {
        re += p[(int64_t)c * nm];
        if (cv == 2) im += p[(int64_t)c * nm + 1];
      }
    } else {   // an invalid entry yields NaN (the host checks its inputs)
      re = im = __longlong_as_double(0x7FF8000000000000ll);
    }
    if (D.complex_output) {
      out[2 * (int64_t)e] = re;
      out[2 * (int64_t)e + 1] = im;
    } else {
      out[e] = re;
    }
  }
}

template <int DIM, int Q, bool CPLX>
cudaError_t launch_group(const DuffyGroupArgs &A, int64_t cap, cudaStream_t s) {
  const size_t smem = sizeof(double) * (size_t)group_smem_doubles<DIM, Q, CPLX>(A.d.n_reg);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  cudaError_t e = cudaSuccess;
  if (smem > 48 * 1024)
    e = cudaFuncSetAttribute(duffy_group_kernel<DIM, Q, CPLX>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int64_t n_work = (int64_t)A.n_groups * A.n_chunks;
  const int64_t grid = std::min<int64_t>(std::min(n_work, cap > 0 ? cap : n_work), 0x7FFFFFFF);
  duffy_group_kernel<DIM, Q, CPLX><<<(unsigned)grid, kGroupThreads, smem, s>>>(A);
  return cudaGetLastError();
}

// the instances: q up to 6 in 3D (5 with complex values: U of a thread is
// q^2 values in registers), up to 8 in 2D
using GroupLaunch = cudaError_t (*)(const DuffyGroupArgs &, int64_t, cudaStream_t);
GroupLaunch group_launch(int dim, int q, bool cplx) {
#define VL1_G(DIM, Q)                                        \
  if (dim == DIM && q == Q)                                  \
    return cplx ? launch_group<DIM, Q, true> : launch_group<DIM, Q, false>;
  VL1_G(2, 1) VL1_G(2, 2) VL1_G(2, 3) VL1_G(2, 4) VL1_G(2, 5) VL1_G(2, 6) VL1_G(2, 7) VL1_G(2, 8)
  VL1_G(3, 1) VL1_G(3, 2) VL1_G(3, 3) VL1_G(3, 4) VL1_G(3, 5)
#undef VL1_G
  if (dim == 3 && q == 6 && !cplx) return launch_group<3, 6, false>;
  return nullptr;
}

}  // namespace
}  // namespace vl1

using namespace vl1;

extern "C" int32_t vl1_duffy_table(const vl1_duffy_desc *desc, double *result, void *stream) {
  if (!desc || !result) {
    set_error("vl1_duffy_table: null descriptor or result");
    return VL1_E_ARG;
  }
  const vl1_duffy_desc &D = *desc;
  if (D.dim < 2 || D.dim > 3 || D.q < 1 || D.q > kDuffyMaxQ || D.n_entries < 0 ||
      D.n_reg < 1 || D.n_rad < 1 || !(D.extent > 0.0) || D.kernel < 0 ||
      D.kernel > VL1_DUFFY_POWER_LOG) {
    set_error("vl1_duffy_table: dim %d, q %d, entries %d, rules %d/%d, extent %g or kernel %d "
              "out of range", D.dim, D.q, D.n_entries, D.n_reg, D.n_rad, D.extent, D.kernel);
    return VL1_E_ARG;
  }
  if (D.derivative != 0 &&
      (D.derivative > D.dim || D.derivative < -D.dim || D.kernel > VL1_DUFFY_HELMHOLTZ3D)) {
    set_error("vl1_duffy_table: derivative %d of kernel %d not supported (Laplace and "
              "Helmholtz first derivatives along an axis)", D.derivative, D.kernel);
    return VL1_E_ARG;
  }
  if ((D.kernel == VL1_DUFFY_POWER && (D.power < 0 || D.power > 64)) ||
      (D.kernel == VL1_DUFFY_POWER_LOG && (D.power < 1 || D.power > 64))) {
    set_error("vl1_duffy_table: power %d out of range for kernel %d", D.power, D.kernel);
    return VL1_E_ARG;
  }
  if (D.n_entries == 0) return VL1_OK;
  if (!D.target_points || !D.decomposition_targets || !D.mode_axes || !D.regular_nodes ||
      !D.regular_weights || !D.radial_nodes || !D.radial_weights || !D.interp_nodes ||
      !D.interp_weights) {
    set_error("vl1_duffy_table: null array in the descriptor");
    return VL1_E_ARG;
  }
  DuffyArgs A;
  A.d = D;
  A.n_perm = D.dim == 3 ? 6 : 2;
  A.n_reg_tail = D.dim == 3 ? D.n_reg * D.n_reg : D.n_reg;
  A.n_sub = 1 << D.dim;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // partial sums per (entry, chunk): stream-ordered scratch, so that a build
  // never waits for work on other streams
  const int n_chunks = A.n_sub * A.n_perm;
  void *scratch = nullptr;
  cudaError_t e = lib_malloc_async(&scratch, sizeof(double) * 2 * (size_t)D.n_entries * n_chunks, s);
  if (e != cudaSuccess) return cuda_fail(e, "allocation of the Duffy partial sums");
  A.part = static_cast<double *>(scratch);
  A.n_chunks = n_chunks;
  // one CTA per (entry, chunk), or at most max_ctas CTAs striding over them
  // (a build that must leave most SMs to other work)
  const int64_t n_work = (int64_t)D.n_entries * n_chunks;
  const int64_t cap = D.max_ctas > 0 ? D.max_ctas : n_work;
  const dim3 grid((unsigned)std::min<int64_t>(std::min(n_work, cap), 0x7FFFFFFF));
  if (D.dim == 3)
    duffy_entry_kernel<3><<<grid, kDuffyThreads, 0, s>>>(A);
  else
    duffy_entry_kernel<2><<<grid, kDuffyThreads, 0, s>>>(A);
  e = cudaGetLastError();
  if (e == cudaSuccess) {
    const int blocks = (int)std::min<int64_t>(((int64_t)D.n_entries + 255) / 256, 4096);
    duffy_reduce_kernel<<<blocks, 256, 0, s>>>(A.part, D.n_entries, n_chunks, D.complex_output,
                                               result);
    e = cudaGetLastError();
  }
  cudaFreeAsync(scratch, s);
  return e == cudaSuccess ? VL1_OK : cuda_fail(e, "duffy_entry_kernel launch");
}

extern "C" int32_t vl1_duffy_table_grouped(const vl1_duffy_desc *desc, int32_t n_groups,
                                           const int32_t *entry_group,
                                           const int32_t *group_entry, double *result,
                                           void *stream) {
  if (!desc || !result || n_groups < 0) {
    set_error("vl1_duffy_table_grouped: null descriptor or result, or n_groups < 0");
    return VL1_E_ARG;
  }
  const vl1_duffy_desc &D = *desc;
  const bool cplx = D.kernel == VL1_DUFFY_HELMHOLTZ2D || D.kernel == VL1_DUFFY_HELMHOLTZ3D;
  const GroupLaunch launch = group_launch(D.dim, D.q, cplx);
  // what the group kernel does not take, and every invalid descriptor, is the
  // per-entry build's
  if (!launch || n_groups == 0 || !entry_group || !group_entry || D.derivative != 0 ||
      D.kernel == VL1_DUFFY_PLANE_WAVE || D.kernel < 0 || D.kernel > VL1_DUFFY_POWER_LOG ||
      D.n_entries < 1 || D.n_reg < 1 || D.n_reg > 128 || D.n_rad < 1 || !(D.extent > 0.0) ||
      (D.kernel == VL1_DUFFY_POWER && (D.power < 0 || D.power > 64)) ||
      (D.kernel == VL1_DUFFY_POWER_LOG && (D.power < 1 || D.power > 64)) ||
      !D.target_points || !D.decomposition_targets || !D.mode_axes || !D.regular_nodes ||
      !D.regular_weights || !D.radial_nodes || !D.radial_weights || !D.interp_nodes ||
      !D.interp_weights)
    return vl1_duffy_table(desc, result, stream);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  DuffyGroupArgs A;
  A.d = D;
  A.n_groups = n_groups;
  A.n_perm = D.dim == 3 ? 6 : 2;
  A.n_chunks = (1 << D.dim) * A.n_perm;
  A.group_entry = group_entry;
  const int cv = cplx ? 2 : 1;
  const int64_t nm = (int64_t)(D.dim == 3 ? D.q * D.q * D.q : D.q * D.q) * cv;
  void *scratch = nullptr;
  cudaError_t e =
      lib_malloc_async(&scratch, sizeof(double) * (size_t)(n_groups * A.n_chunks * nm), s);
  if (e != cudaSuccess) return cuda_fail(e, "allocation of the Duffy partial sums");
  A.part = static_cast<double *>(scratch);
  e = launch(A, D.max_ctas, s);
  if (e == cudaSuccess) {
    const int blocks = (int)std::min<int64_t>(((int64_t)D.n_entries + 127) / 128, 4096);
    duffy_group_reduce_kernel<<<blocks, 128, 0, s>>>(D, A.part, entry_group, A.n_chunks, cv,
                                                    result);
    e = cudaGetLastError();
  }
  cudaFreeAsync(scratch, s);
  return e == cudaSuccess ? VL1_OK : cuda_fail(e, "duffy_group_kernel launch");
}
