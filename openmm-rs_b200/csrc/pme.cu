// PME reciprocal space (forces/pme.rs:141-425): order-5 cardinal B-spline spreading of the
// charges, 3-D FFT (cuFFT, real-to-complex), multiplication by the influence function, inverse
// FFT and force gather.
//
// The reference transforms the full complex grid; here the charge grid is real, so the
// forward transform is R2C and only the kz <= nz/2 half is stored.  The influence table holds
// 0.5 * (G(m) + G(m')) for each stored element m and its conjugate partner m' (the reference's
// mode numbering makes them differ only on Nyquist planes of triclinic boxes), which is exactly
// what the reference's "real part of the inverse transform" keeps.  The energy is
// 0.5 * sum_full G |S|^2 = sum_half w * 0.5 * G_sym |S|^2 with w = 1 on the kz = 0 and
// kz = nz/2 planes and 2 elsewhere.
//
// Charges are spread into a 64-bit fixed-point grid (units of 2^-40 e) so the grid, and every
// force derived from it, is independent of the order of the atomic additions.
#include <cooperative_groups.h>

#include "kernels.h"

namespace ommb200 {
namespace {

namespace cg = cooperative_groups;

// pme.rs:151-174
template <class Real>
__device__ __forceinline__ void spline5(Real f, Real w[5], Real dw[5]) {
  w[0] = Real(1) - f;
  w[1] = f;
  w[2] = w[3] = w[4] = Real(0);
#pragma unroll
  for (int order = 3; order <= 5; ++order) {
    if (order == 5) {
      dw[0] = -w[0];
#pragma unroll
      for (int i = 1; i < 5; ++i) dw[i] = w[i - 1] - w[i];
    }
    const Real inv = Real(1) / Real(order - 1);
    w[order - 1] = f * w[order - 2] * inv;
#pragma unroll
    for (int i = order - 2; i >= 1; --i)
      w[i] = ((f + Real(order - 1 - i)) * w[i - 1] + (Real(i + 1) - f) * w[i]) * inv;
    w[0] *= (Real(1) - f) * inv;
  }
}

// pme.rs:201-218: base grid index and fraction along each axis, in f64.  Returns false for a
// nonfinite position, which then touches no grid point (the integrator reports it).
template <class Real>
__device__ __forceinline__ bool stencil(const PmeArgs<Real>& a, int atom, int base[3],
                                        Real frac[3]) {
  const double x = a.pos[3 * atom], y = a.pos[3 * atom + 1], z = a.pos[3 * atom + 2];
  const int dims[3] = {a.nx, a.ny, a.nz};
  bool ok = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double f = x * a.recip[d][0] + y * a.recip[d][1] + z * a.recip[d][2];
    const double coord = (f - floor(f)) * (double)dims[d];
    ok = ok && coord >= 0.0 && coord <= (double)dims[d];
    const double fl = ok ? floor(coord) : 0.0;
    const int b = (int)fl;
    base[d] = (unsigned)b < (unsigned)dims[d] ? b : 0;  // fl may round up to dims
    frac[d] = (Real)(ok ? coord - fl : 0.0);
  }
  return ok;
}
// The particle in place s of the visiting order (which of its two copies is the same for every
// thread of the launch: nothing beside it writes the parity), -1 for padding.
template <class Real>
__device__ __forceinline__ int ordered_atom(const PmeArgs<Real>& a, int s) {
  if (s >= a.n_order) return -1;
  if (!a.order) return s;
  return a.order[a.order_parity ? (size_t)*a.order_parity * a.n_order + s : s];
}
template <class Real>
__global__ void spread_kernel(const PmeArgs<Real> a) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const int atom = ordered_atom(a, s);
  if (atom < 0) return;
  const double qd = a.charge[atom];
  if (qd == 0.0) return;
  const Real q = (Real)qd;
  int base[3];
  Real frac[3], w[3][5], dw[3][5];
  if (!stencil(a, atom, base, frac)) return;
#pragma unroll
  for (int d = 0; d < 3; ++d) spline5(frac[d], w[d], dw[d]);
  const Real gscale = Real(kGridScale);
  for (int ix = 0; ix < 5; ++ix) {
    int gx = base[0] + ix;
    gx -= gx >= a.nx ? a.nx : 0;
    const Real qx = q * w[0][ix];
    for (int iy = 0; iy < 5; ++iy) {
      int gy = base[1] + iy;
      gy -= gy >= a.ny ? a.ny : 0;
      const Real qxy = qx * w[1][iy];
      long long* row = a.grid_fixed + ((long long)gx * a.ny + gy) * a.nz;
#pragma unroll
      for (int iz = 0; iz < 5; ++iz) {
        int gz = base[2] + iz;
        gz -= gz >= a.nz ? a.nz : 0;
        add_fixed(row + gz, to_fixed(qxy * w[2][iz], gscale));
      }
    }
  }
}

// Staged spreading: a CTA takes 64 consecutive sorted slots (spatially compact: part of one
// x-y column, z-sorted), two threads per atom, and adds the atoms' 125-point stencils into a
// shared-memory copy of the grid box they touch, then adds that box to the global grid, so
// each grid point receives one global atomic per CTA instead of one per stencil.  Shared
// accumulation uses native 32-bit integer atomics (64-bit shared atomics measured 1.5-1.8x
// slower).  FP64 form: a split of each 2^-40 fixed-point value, v = hi 2^20 + lo with
// 0 <= lo < 2^20; at most 64 contributions per cell keep both partial sums inside 32 bits (for
// |q| < 16 e), and hi_sum 2^20 + lo_sum recovers the exact 64-bit total.  FP32 form: one atomic
// per point, each contribution (a float product) rounded to 2^-26 e, which keeps 64 of them
// inside 32 bits for |q| < 2 e (the order-5 B-spline peaks at 115/192 per axis, so a point gets
// at most 0.22 |q| from an atom); the box is added to the 2^-40 global grid scaled by 2^14,
// exactly.  Either way the sums are exact integers, so the grid does not depend on the order
// of the additions; nor on how the particles are grouped into CTAs: a CTA whose box exceeds
// kSpreadCells (it straddles a periodic edge of the column order) spreads directly with the same
// rounding, and a particle of larger charge spreads directly at 2^-40 e wherever it is.
constexpr int kSpreadAtoms = 64;
constexpr int kSpreadCells = 4096;
constexpr float kSpreadScale32 = 67108864.f;           // 2^26 (FP32 form, staged)
constexpr long long kSpreadWiden32 = 1ll << 14;        // 2^40 / 2^26

template <class Real>
__global__ void __launch_bounds__(2 * kSpreadAtoms) spread_staged_kernel(const PmeArgs<Real> a) {
  __shared__ int c_hi[kSpreadCells];
  __shared__ unsigned int c_lo[kSpreadCells];
  __shared__ int s_lo[3], s_hi[3];
  const int tid = threadIdx.x, half = tid / kSpreadAtoms;  // half 0: ix 0..2, half 1: ix 3..4
  const int s = blockIdx.x * kSpreadAtoms + (tid % kSpreadAtoms);
  const int atom = ordered_atom(a, s);
  const double qd = atom >= 0 ? a.charge[atom] : 0.0;
  int base[3] = {0, 0, 0};
  Real frac[3] = {Real(0), Real(0), Real(0)};
  const bool ok = atom >= 0 && qd != 0.0 && stencil(a, atom, base, frac);
  // the 32-bit partial sums need |q| < 2 e (FP32 form) or |q| < 16 e (FP64 form)
  const bool big = ok && fabs(qd) >= (sizeof(Real) == 4 ? 2.0 : 16.0), staged = ok && !big;
  if (tid < 3) {
    s_lo[tid] = 0x7fffffff;
    s_hi[tid] = -1;
  }
  __syncthreads();
  if (staged && half == 0) {
    for (int d = 0; d < 3; ++d) {
      atomicMin(&s_lo[d], base[d]);
      atomicMax(&s_hi[d], base[d]);
    }
  }
  __syncthreads();
  const int lo0 = s_lo[0], lo1 = s_lo[1], lo2 = s_lo[2];
  const int ex = s_hi[0] - lo0 + 5, ey = s_hi[1] - lo1 + 5, ez = s_hi[2] - lo2 + 5;
  const bool any = s_hi[0] >= 0;
  const long long n_cells = any ? (long long)ex * ey * ez : 0;
  Real w[3][5], dw[3][5];
  if (ok) {
#pragma unroll
    for (int d = 0; d < 3; ++d) spline5(frac[d], w[d], dw[d]);
  }
  const Real q = (Real)qd;
  const Real gscale = Real(kGridScale);
  const int ix0 = half == 0 ? 0 : 3, ix1 = half == 0 ? 3 : 5;
  if (big || (staged && n_cells > kSpreadCells)) {  // direct spreading
    for (int ix = ix0; ix < ix1; ++ix) {
      int gx = base[0] + ix;
      gx -= gx >= a.nx ? a.nx : 0;
      const Real qx = q * w[0][ix];
      for (int iy = 0; iy < 5; ++iy) {
        int gy = base[1] + iy;
        gy -= gy >= a.ny ? a.ny : 0;
        const Real qxy = qx * w[1][iy];
        long long* row = a.grid_fixed + ((long long)gx * a.ny + gy) * a.nz;
#pragma unroll
        for (int iz = 0; iz < 5; ++iz) {
          int gz = base[2] + iz;
          gz -= gz >= a.nz ? a.nz : 0;
          // rounded as the particle's staged contributions are, whatever CTA it is in, so the
          // grid does not depend on the visiting order
          long long v;
          if (sizeof(Real) == 4 && !big)
            v = (long long)__float2int_rn((float)(qxy * w[2][iz]) * kSpreadScale32) * kSpreadWiden32;
          else
            v = to_fixed(qxy * w[2][iz], gscale);
          add_fixed(row + gz, v);
        }
      }
    }
  }
  if (!any || n_cells > kSpreadCells) return;  // uniform
  const int nc = (int)n_cells;
  for (int c = tid; c < nc; c += 2 * kSpreadAtoms) {
    c_hi[c] = 0;
    if constexpr (sizeof(Real) == 8) c_lo[c] = 0u;
  }
  __syncthreads();
  if (staged) {
    for (int ix = ix0; ix < ix1; ++ix) {
      const Real qx = q * w[0][ix];
      for (int iy = 0; iy < 5; ++iy) {
        const Real qxy = qx * w[1][iy];
        const int row = ((base[0] - lo0 + ix) * ey + (base[1] - lo1 + iy)) * ez + (base[2] - lo2);
#pragma unroll
        for (int iz = 0; iz < 5; ++iz) {
          if constexpr (sizeof(Real) == 4) {
            atomicAdd(&c_hi[row + iz], __float2int_rn(qxy * w[2][iz] * kSpreadScale32));
          } else {
            const long long v = to_fixed(qxy * w[2][iz], gscale);
            atomicAdd(&c_hi[row + iz], (int)(v >> 20));
            atomicAdd(&c_lo[row + iz], (unsigned int)(v & 0xFFFFF));
          }
        }
      }
    }
  }
  __syncthreads();
  for (int c = tid; c < nc; c += 2 * kSpreadAtoms) {
    const long long v = sizeof(Real) == 4 ? (long long)c_hi[c] * kSpreadWiden32
                                          : (long long)c_hi[c] * (1ll << 20) + (long long)c_lo[c];
    if (v == 0) continue;
    const int cz = c % ez, cy = (c / ez) % ey, cx = c / (ez * ey);
    int gx = lo0 + cx, gy = lo1 + cy, gz = lo2 + cz;
    gx -= gx >= a.nx ? a.nx : 0;
    gy -= gy >= a.ny ? a.ny : 0;
    gz -= gz >= a.nz ? a.nz : 0;
    add_fixed(a.grid_fixed + ((long long)gx * a.ny + gy) * a.nz + gz, v);
  }
}

template <class Real>
__global__ void convert_kernel(const PmeArgs<Real> a) {
  const long long total = (long long)a.nx * a.ny * a.nz;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    a.grid_real[i] = (Real)((double)a.grid_fixed[i] * kGridScaleInv);
    a.grid_fixed[i] = 0;
  }
}

template <class Real>
struct Cplx;
template <>
struct Cplx<float> {
  using T = float2;
};
template <>
struct Cplx<double> {
  using T = double2;
};

__device__ __forceinline__ double freq(int k, int n) { return k < (n + 1) / 2 ? (double)k : (double)(k - n); }

// Reciprocal-space energy and virial of half-spectrum element (x, y, z) with |S|^2 = s2 and
// influence value infl (pme.rs:307-372): the element and its conjugate partner each carry
// half of the virial, elements with 0 < z < nz/2 count twice.
template <int kTerms, class Real>
__device__ __forceinline__ void mode_energy(const PmeArgs<Real>& a, int x, int y, int z, double s2,
                                            double infl, double& e, double (&w)[6]) {
  const double wz = (z == 0 || (a.nz % 2 == 0 && z == a.nz / 2)) ? 1.0 : 2.0;
  e += wz * 0.5 * infl * s2;
  if (kTerms == kTermsEnergy) return;
  const int idx[2][3] = {{x, y, z}, {(a.nx - x) % a.nx, (a.ny - y) % a.ny, (a.nz - z) % a.nz}};
  for (int p = 0; p < 2; ++p) {
    const double m[3] = {freq(idx[p][0], a.nx), freq(idx[p][1], a.ny), freq(idx[p][2], a.nz)};
    double k[3];
    for (int c = 0; c < 3; ++c) k[c] = m[0] * a.recip[0][c] + m[1] * a.recip[1][c] + m[2] * a.recip[2][c];
    const double k2 = k[0] * k[0] + k[1] * k[1] + k[2] * k[2];
    const double bm = a.moduli[idx[p][0]] * a.moduli[a.nx + idx[p][1]] * a.moduli[a.nx + a.ny + idx[p][2]];
    const double pa = kPiD * kPiD / (a.alpha * a.alpha);
    const double g_m = kOne4PiEps0 * exp(-pa * k2) / (kPiD * a.volume * k2 * bm);
    const double em = wz * 0.5 * 0.5 * g_m * s2;
    const double c = 2.0 * (1.0 + pa * k2) / k2;
    w[0] += em * (1.0 - c * k[0] * k[0]);
    w[1] += em * (1.0 - c * k[1] * k[1]);
    w[2] += em * (1.0 - c * k[2] * k[2]);
    w[3] -= em * c * k[0] * k[1];
    w[4] -= em * c * k[0] * k[2];
    w[5] -= em * c * k[1] * k[2];
  }
}

// The CTA's sums in fixed point (every thread of the block calls it).
template <int kTerms, class Real>
__device__ __forceinline__ void commit_energy(const PmeArgs<Real>& a, double e, const double (&w)[6]) {
  long long ef = to_fixed(e, kEnergyScale);
  long long wf[6] = {0, 0, 0, 0, 0, 0};
  if (kTerms > kTermsEnergy)
    for (int c = 0; c < 6; ++c) wf[c] = to_fixed(w[c], kEnergyScale);
  for (int off = 16; off > 0; off >>= 1) {
    ef += __shfl_xor_sync(0xffffffffu, ef, off);
    if (kTerms > kTermsEnergy)
      for (int c = 0; c < 6; ++c) wf[c] += __shfl_xor_sync(0xffffffffu, wf[c], off);
  }
  commit_cta<kTerms>(a.energy, ef, wf);
}

template <class Real, int kTerms>
__global__ void convolve_kernel(const PmeArgs<Real> a) {
  using C2 = typename Cplx<Real>::T;
  C2* g = reinterpret_cast<C2*>(a.grid_k);
  const int nzh = a.nz / 2 + 1;
  const long long total = (long long)a.nx * a.ny * nzh;
  double e = 0.0, w[6] = {0, 0, 0, 0, 0, 0};
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    C2 v = g[i];
    const Real infl = a.influence[i];
    if (kTerms && i != 0) {
      const int z = (int)(i % nzh);
      const int y = (int)((i / nzh) % a.ny);
      const int x = (int)(i / ((long long)nzh * a.ny));
      mode_energy<kTerms>(a, x, y, z, (double)v.x * v.x + (double)v.y * v.y, (double)infl, e, w);
    }
    v.x *= infl;
    v.y *= infl;
    g[i] = v;
  }
  if (kTerms) commit_energy<kTerms>(a, e, w);
}

// pme.rs:377-425.  Eight lanes per atom: lane k < 5 sums the 25 grid points of stencil plane
// ix = k, then the group reduces by a fixed shuffle tree and lane 0 commits the force.
template <class Real>
__global__ void gather_kernel(const PmeArgs<Real> a) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int s = t >> 3, k = t & 7;
  const int atom = ordered_atom(a, s);
  const double qd = atom >= 0 ? a.charge[atom] : 0.0;
  int base[3] = {0, 0, 0};
  Real frac[3] = {Real(0), Real(0), Real(0)};
  const bool ok = atom >= 0 && qd != 0.0 && stencil(a, atom, base, frac);
  Real g0 = 0, g1 = 0, g2 = 0;
  if (ok && k < 5) {
    Real w[3][5], dw[3][5];
#pragma unroll
    for (int d = 0; d < 3; ++d) spline5(frac[d], w[d], dw[d]);
    int gx = base[0] + k;
    gx -= gx >= a.nx ? a.nx : 0;
    Real wx = w[0][0], dwx = dw[0][0];
#pragma unroll
    for (int i = 1; i < 5; ++i)
      if (k == i) {
        wx = w[0][i];
        dwx = dw[0][i];
      }
    for (int iy = 0; iy < 5; ++iy) {
      int gy = base[1] + iy;
      gy -= gy >= a.ny ? a.ny : 0;
      const Real* row = a.grid_real + ((long long)gx * a.ny + gy) * a.nz;
      const Real wxy = wx * w[1][iy];
      const Real dxy = dwx * w[1][iy];
      const Real xdy = wx * dw[1][iy];
#pragma unroll
      for (int iz = 0; iz < 5; ++iz) {
        int gz = base[2] + iz;
        gz -= gz >= a.nz ? a.nz : 0;
        const Real phi = row[gz];
        g0 += phi * dxy * w[2][iz];
        g1 += phi * xdy * w[2][iz];
        g2 += phi * wxy * dw[2][iz];
      }
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    g0 += __shfl_xor_sync(0xffffffffu, g0, o, 8);
    g1 += __shfl_xor_sync(0xffffffffu, g1, o, 8);
    g2 += __shfl_xor_sync(0xffffffffu, g2, o, 8);
  }
  if (!ok || k != 0) return;
  const double gd[3] = {(double)g0 * a.nx, (double)g1 * a.ny, (double)g2 * a.nz};
  for (int c = 0; c < 3; ++c) {
    const double f = -qd * (gd[0] * a.recip[0][c] + gd[1] * a.recip[1][c] + gd[2] * a.recip[2][c]);
    add_fixed(a.force + (long long)c * a.n_atoms + atom, to_fixed(f, kForceScale));
  }
}

// ---- own 3-D transform of the PME grid -------------------------------------------------
// Replaces the fixed-point conversion, the real-to-complex / complex-to-real cuFFT pair and
// the convolution by three kernels over the half spectrum [x][y][kz <= nz/2]:
//   planes_forward  one CTA per x plane: fixed-point grid -> real (grid zeroed), z transform
//                   of two real rows at once as one complex row, y transform
//   x_convolve      one CTA per (y, run of kz): x transform, influence function (+ energy
//                   and virial), inverse x transform
//   planes_inverse  one CTA per x plane: inverse y transform, inverse z transform of two
//                   Hermitian rows at once, real rows -> potential grid for the gather
// Every 1-D transform is a mixed-radix Stockham FFT in shared memory (radices 2, 3, 4, 5, 7,
// 8; one radix-R butterfly per thread and stage; one larger prime as the first stage, by direct
// sums), forward sign exp(-2 pi i jk/n) and unnormalised like cuFFT; the inverse is
// conj(F(conj(x))).  Sizes with other prime factors use cuFFT.
template <class C2>
__device__ __forceinline__ C2 cmul(C2 a, C2 w) {
  C2 r;
  r.x = a.x * w.x - a.y * w.y;
  r.y = a.x * w.y + a.y * w.x;
  return r;
}
template <class C2>
__device__ __forceinline__ C2 conjg(C2 a) {
  a.y = -a.y;
  return a;
}
template <class C2>
__device__ __forceinline__ void bfly2(C2& a, C2& b) {
  const C2 t = a;
  a.x = t.x + b.x;
  a.y = t.y + b.y;
  b.x = t.x - b.x;
  b.y = t.y - b.y;
}
// multiplication by -i
template <class C2>
__device__ __forceinline__ C2 mul_mi(C2 a) {
  C2 r;
  r.x = a.y;
  r.y = -a.x;
  return r;
}
template <class C2>
__device__ __forceinline__ void dft4(C2& a0, C2& a1, C2& a2, C2& a3) {
  bfly2(a0, a2);  // a0 = x0 + x2, a2 = x0 - x2
  bfly2(a1, a3);  // a1 = x1 + x3, a3 = x1 - x3
  a3 = mul_mi(a3);
  bfly2(a0, a1);  // y0, y2
  bfly2(a2, a3);  // y1, y3
  const C2 y1 = a2, y2 = a1;
  a1 = y1;
  a2 = y2;
}

// Forward DFT of R values in registers.  Radices 2, 4, 8 use butterflies; the odd primes use
// the direct sum with W_R^q = tw[q n / R] from the length-n twiddle table.
template <int R, class C2>
__device__ __forceinline__ void dft_reg(C2 (&v)[R], const C2* tw, int n) {
  using S = decltype(v[0].x);
  if constexpr (R == 2) {
    bfly2(v[0], v[1]);
  } else if constexpr (R == 4) {
    dft4(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 8) {
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    const S h = (S)0.70710678118654752440;  // 1/sqrt(2)
    C2 o1, o2, o3;
    o1.x = h * (v[3].x + v[3].y);  // W_8 = (1 - i)/sqrt(2)
    o1.y = h * (v[3].y - v[3].x);
    o2 = mul_mi(v[5]);              // W_8^2 = -i
    o3.x = h * (v[7].y - v[7].x);  // W_8^3 = -(1 + i)/sqrt(2)
    o3.y = -h * (v[7].x + v[7].y);
    C2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], d0 = v[1];
    bfly2(e0, d0);
    bfly2(e1, o1);
    bfly2(e2, o2);
    bfly2(e3, o3);
    v[0] = e0; v[4] = d0;
    v[1] = e1; v[5] = o1;
    v[2] = e2; v[6] = o2;
    v[3] = e3; v[7] = o3;
  } else {
    const int st = n / R;
    C2 out[R];
#pragma unroll
    for (int s = 0; s < R; ++s) {
      C2 acc = v[0];
#pragma unroll
      for (int q = 1; q < R; ++q) {
        const C2 w = tw[((q * s) % R) * st];
        acc.x += v[q].x * w.x - v[q].y * w.y;
        acc.y += v[q].x * w.y + v[q].y * w.x;
      }
      out[s] = acc;
    }
#pragma unroll
    for (int s = 0; s < R; ++s) v[s] = out[s];
  }
}

// One Stockham stage over P pencils of length n (pencil p at in + p n): butterfly j of a
// pencil reads in[j + r n/R], applies the twiddles W_n^(r k n/(ns R)) of its position
// k = j mod ns in the current sub-transforms of length ns, and writes out[(j/ns) ns R + k + r ns].
// Not inlined: every transform of a kernel shares one copy of each radix's code, which keeps
// the instruction footprint of a CTA (one CTA per SM, every stage a new code path) small.
template <int R, class C2>
__device__ __noinline__ void stockham_stage(const C2* in, C2* out, const C2* tw, int n, int ns, int P) {
  const int nr = n / R, items = P * nr, span = n / (ns * R);
  for (int t = threadIdx.x; t < items; t += blockDim.x) {
    const int p = t / nr, j = t - p * nr, q = j / ns, k = j - q * ns;
    const C2* src = in + p * n + j;
    C2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[r * nr];
    if (ns > 1) {
      const int step = k * span;
#pragma unroll
      for (int r = 1; r < R; ++r) v[r] = cmul(v[r], tw[r * step]);
    }
    dft_reg<R>(v, tw, n);
    C2* dst = out + p * n + q * ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) dst[r * ns] = v[r];
  }
}

// First stage (ns = 1) for a prime radix R > 7: outputs m and R - m of a sub-transform are the
// sum and difference of the same four real sums over its R inputs, so a thread that owns both
// spends 4 multiply-adds and two shared loads (one of them a broadcast: the lanes of a warp
// mostly share their inputs) per input instead of 8 and four.
template <class C2>
__device__ __noinline__ void stockham_prime(const C2* in, C2* out, const C2* tw, int n, int R, int P) {
  using S = decltype(in->x);
  const int nr = n / R, nh = (R + 1) / 2, items = P * nr * nh;
  for (int t = threadIdx.x; t < items; t += blockDim.x) {
    const int pj = t / nh, m = t - pj * nh, p = pj / nr, j = pj - p * nr;
    const C2* src = in + p * n + j;
    C2* dst = out + p * n + j * R;
    const C2 v0 = src[0];
    S xc = v0.x, yc = v0.y, xs = 0, ys = 0;  // sums of x cos, y cos, x sin, y sin
    const int step = m * nr;
    int w = 0;
#pragma unroll 4
    for (int r = 1; r < R; ++r) {
      w += step;
      w -= w >= n ? n : 0;
      const C2 v = src[r * nr], e = tw[w];  // e = (cos, -sin)
      xc += v.x * e.x;
      yc += v.y * e.x;
      xs += v.x * e.y;
      ys += v.y * e.y;
    }
    C2 a, b;
    a.x = xc - ys;
    a.y = yc + xs;
    b.x = xc + ys;
    b.y = yc - xs;
    dst[m] = a;
    if (m) dst[R - m] = b;
  }
}

// Forward transform of P pencils held in a (b: scratch of the same size); returns the buffer
// that holds the result.  The callers synchronise before and after.
template <class C2>
__device__ C2* stockham(C2* a, C2* b, const C2* tw, const PmeFft& f, int axis, int n, int P) {
  int ns = 1;
  for (int s = 0; s < f.nrad[axis]; ++s) {
    const int R = f.rad[axis][s];
    switch (R) {
      case 2: stockham_stage<2>(a, b, tw, n, ns, P); break;
      case 3: stockham_stage<3>(a, b, tw, n, ns, P); break;
      case 4: stockham_stage<4>(a, b, tw, n, ns, P); break;
      case 5: stockham_stage<5>(a, b, tw, n, ns, P); break;
      case 7: stockham_stage<7>(a, b, tw, n, ns, P); break;
      case 8: stockham_stage<8>(a, b, tw, n, ns, P); break;
      default: stockham_prime(a, b, tw, n, R, P); break;  // always the first stage
    }
    __syncthreads();
    C2* t = a;
    a = b;
    b = t;
    ns *= R;
  }
  return a;
}

template <class C2>
__device__ __forceinline__ void load_twiddles(C2* dst, const void* src, int n) {
  const C2* t = reinterpret_cast<const C2*>(src);
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = t[i];
}

// Shared memory of a plane kernel: z and y twiddles, two buffers of `plane` elements.
__host__ __device__ inline int fft_plane_elems(int ny, int nz) {
  const int a = (ny + 1) / 2 * nz, b = (nz / 2 + 1) * ny;
  return a > b ? a : b;
}

constexpr int kPlaneThreads = 512, kXPassThreads = 256;  // block size caps of the transform
constexpr int kClusterThreads = 512;
constexpr int kLoadBatch = 4;  // global loads each thread keeps in flight in the copy loops

// for i in [0, total), strided over the block: v = load(i) for kLoadBatch items at a time,
// then use(i, v) for each, so that the loads of a batch overlap.
template <class T, class Load, class Use>
__device__ __forceinline__ void batched(int total, Load load, Use use) {
  for (int i0 = threadIdx.x; i0 < total; i0 += kLoadBatch * blockDim.x) {
    T v[kLoadBatch];
#pragma unroll
    for (int u = 0; u < kLoadBatch; ++u) {
      const int i = i0 + u * blockDim.x;
      if (i < total) v[u] = load(i);
    }
#pragma unroll
    for (int u = 0; u < kLoadBatch; ++u) {
      const int i = i0 + u * blockDim.x;
      if (i < total) use(i, v[u]);
    }
  }
}

template <class Real>
__global__ void __launch_bounds__(kPlaneThreads) planes_forward(const PmeArgs<Real> a, const PmeFft f) {
  using C2 = typename Cplx<Real>::T;
  extern __shared__ __align__(16) unsigned char fsm[];
  const int ny = a.ny, nz = a.nz, nzh = nz / 2 + 1, nyp = (ny + 1) / 2, x = blockIdx.x;
  const int pe = fft_plane_elems(ny, nz);
  C2* twz = reinterpret_cast<C2*>(fsm);
  C2* twy = twz + nz;
  C2* A = twy + ny;
  C2* B = A + pe;
  load_twiddles(twz, f.tw[2], nz);
  load_twiddles(twy, f.tw[1], ny);
  // rows y = 2 yp (real part) and 2 yp + 1 (imaginary part) as one complex row
  long long* plane = a.grid_fixed + (long long)x * ny * nz;
  batched<longlong2>(
      nyp * nz,
      [&](int i) {
        const int yp = i / nz, z = i - yp * nz;
        const long long* g0 = plane + (long long)(2 * yp) * nz + z;
        longlong2 r;
        r.x = __ldcg(g0);
        r.y = 2 * yp + 1 < ny ? __ldcg(g0 + nz) : 0;
        return r;
      },
      [&](int i, longlong2 r) {
        C2 v;
        v.x = (Real)((double)r.x * kGridScaleInv);
        v.y = (Real)((double)r.y * kGridScaleInv);
        A[i] = v;
      });
  __syncthreads();
  for (int i = threadIdx.x; i < ny * nz; i += blockDim.x) plane[i] = 0;  // ready for the next spread
  C2* r = stockham(A, B, twz, f, 2, nz, nyp);
  C2* o = r == A ? B : A;
  // split the two real rows' spectra: X_even = (Z_k + conj Z_-k)/2, X_odd = -i (Z_k - conj Z_-k)/2,
  // into pencils along y: o[kz][y]
  for (int i = threadIdx.x; i < nzh * ny; i += blockDim.x) {
    const int kz = i / ny, y = i - kz * ny, yp = y >> 1;
    const C2 zk = r[yp * nz + kz], zm = r[yp * nz + (kz == 0 ? 0 : nz - kz)];
    C2 v;
    if ((y & 1) == 0) {
      v.x = (Real)0.5 * (zk.x + zm.x);
      v.y = (Real)0.5 * (zk.y - zm.y);
    } else {
      v.x = (Real)0.5 * (zk.y + zm.y);
      v.y = (Real)0.5 * (zm.x - zk.x);
    }
    o[i] = v;
  }
  __syncthreads();
  C2* s = stockham(o, r, twy, f, 1, ny, nzh);
  C2* out = reinterpret_cast<C2*>(a.grid_k) + (long long)x * ny * nzh;
  for (int i = threadIdx.x; i < ny * nzh; i += blockDim.x) {
    const int y = i / nzh, kz = i - y * nzh;
    out[i] = s[kz * ny + y];
  }
}

template <class Real, int kTerms>
__global__ void __launch_bounds__(kXPassThreads) x_convolve(const PmeArgs<Real> a, const PmeFft f) {
  using C2 = typename Cplx<Real>::T;
  extern __shared__ __align__(16) unsigned char fsm[];
  const int nx = a.nx, nzh = a.nz / 2 + 1, P0 = f.pencils_x;
  const int nkb = (nzh + P0 - 1) / P0;
  const int y = blockIdx.x / nkb, kz0 = (blockIdx.x - y * nkb) * P0, P = min(P0, nzh - kz0);
  C2* tw = reinterpret_cast<C2*>(fsm);
  C2* A = tw + nx;
  C2* B = A + P0 * nx;
  load_twiddles(tw, f.tw[0], nx);
  C2* g = reinterpret_cast<C2*>(a.grid_k);
  const long long sx = (long long)a.ny * nzh, base = (long long)y * nzh + kz0;
  batched<C2>(
      nx * P, [&](int i) { const int x = i / P, p = i - x * P; return __ldcg(g + base + x * sx + p); },
      [&](int i, C2 v) { const int x = i / P, p = i - x * P; A[p * nx + x] = v; });
  __syncthreads();
  C2* r = stockham(A, B, tw, f, 0, nx, P);
  C2* o = r == A ? B : A;
  double e = 0.0, w[6] = {0, 0, 0, 0, 0, 0};
  batched<Real>(
      P * nx, [&](int i) { const int p = i / nx, x = i - p * nx; return __ldg(a.influence + base + x * sx + p); },
      [&](int i, Real infl) {
        const int p = i / nx, x = i - p * nx;
        C2 v = r[i];
        if (kTerms && base + x * sx + p != 0)
          mode_energy<kTerms>(a, x, y, kz0 + p, (double)v.x * v.x + (double)v.y * v.y, (double)infl, e, w);
        v.x *= infl;
        v.y *= -infl;  // conjugated for the inverse transform
        r[i] = v;
      });
  if (kTerms) commit_energy<kTerms>(a, e, w);
  __syncthreads();
  C2* s = stockham(r, o, tw, f, 0, nx, P);
  for (int i = threadIdx.x; i < nx * P; i += blockDim.x) {
    const int x = i / P, p = i - x * P;
    g[base + x * sx + p] = conjg(s[p * nx + x]);
  }
}

template <class Real>
__global__ void __launch_bounds__(kPlaneThreads) planes_inverse(const PmeArgs<Real> a, const PmeFft f) {
  using C2 = typename Cplx<Real>::T;
  extern __shared__ __align__(16) unsigned char fsm[];
  const int ny = a.ny, nz = a.nz, nzh = nz / 2 + 1, nyp = (ny + 1) / 2, x = blockIdx.x;
  const int pe = fft_plane_elems(ny, nz);
  C2* twz = reinterpret_cast<C2*>(fsm);
  C2* twy = twz + nz;
  C2* A = twy + ny;
  C2* B = A + pe;
  load_twiddles(twz, f.tw[2], nz);
  load_twiddles(twy, f.tw[1], ny);
  const C2* in = reinterpret_cast<const C2*>(a.grid_k) + (long long)x * ny * nzh;
  batched<C2>(
      ny * nzh, [&](int i) { return __ldcg(in + i); },
      [&](int i, C2 v) { const int y = i / nzh, kz = i - y * nzh; A[kz * ny + y] = conjg(v); });
  __syncthreads();
  // r = F(conj H): the inverse y transform of H is conj(r)
  C2* r = stockham(A, B, twy, f, 1, ny, nzh);
  C2* o = r == A ? B : A;
  // rows 2 yp and 2 yp + 1 of the inverse, Hermitian-completed along z, as one row
  // Z = Ha + i Hb, stored conjugated: conj Z = conj Ha - i conj Hb
  for (int i = threadIdx.x; i < nyp * nz; i += blockDim.x) {
    const int yp = i / nz, k = i - yp * nz, y0 = 2 * yp;
    const bool lo = k < nzh;
    const int kk = lo ? k : nz - k;
    C2 ca = r[kk * ny + y0];  // conj Ha[k] for k < nzh
    if (!lo) ca = conjg(ca);
    C2 cb;
    cb.x = cb.y = 0;
    if (y0 + 1 < ny) {
      cb = r[kk * ny + y0 + 1];
      if (!lo) cb = conjg(cb);
    }
    C2 v;
    v.x = ca.x + cb.y;
    v.y = ca.y - cb.x;
    o[i] = v;
  }
  __syncthreads();
  // s = F(conj Z); the inverse is conj(s): row 2 yp = Re s, row 2 yp + 1 = -Im s
  C2* s = stockham(o, r, twz, f, 2, nz, nyp);
  Real* out = a.grid_real + (long long)x * ny * nz;
  for (int i = threadIdx.x; i < ny * nz; i += blockDim.x) {
    const int y = i / nz, z = i - y * nz;
    const C2 v = s[(y >> 1) * nz + z];
    out[i] = (y & 1) ? -v.y : v.x;
  }
}

// ---- the whole reciprocal part of a small box in one launch -----------------------------
// Below a few thousand particles the five launches of the reciprocal chain (spread, three
// transform passes, gather) are bound by their launches and by one round trip to L2 each; the
// grid itself (23^3 to about 40^3) fits in the shared memory of one thread-block cluster.  CTA c
// of the cluster owns the x planes [c P, (c + 1) P) of the grid from the charges to the
// potential: it spreads every particle's stencil rows that fall in its planes into shared
// memory (exact fixed point at 2^-40 e, split hi 2^20 + lo for native 32-bit atomics: at most
// kClusterAtoms contributions keep lo inside 32 bits, and the host checks sum |q| for hi),
// transforms its planes along z and y, transforms its share of the (y, kz) pencils along x with
// the influence function, reading and writing the owners' planes through distributed shared
// memory, transforms its planes back and gathers their part of every particle's force.  Two
// cluster barriers (around the x pass) replace four kernel boundaries.  Each particle's force
// is the fixed-point sum of its planes' parts.  1,524 particles on a 23^3 grid: a step with the
// chain's launches takes 55 us, with this form 42 (46 when each thread walked its particles'
// whole stencils, spread and gather, instead of a list).
template <class Real>
struct ClusterLayout {  // element counts; every CTA of the cluster has the same
  int planes, pencils;  // planes and x pencils per CTA
  size_t plane_elems;   // of each of the two plane buffers
  int list;             // capacity of the particle list
  __host__ __device__ ClusterLayout(int nx, int ny, int nz, int ctas, int list_capacity)
      : planes((nx + ctas - 1) / ctas), pencils((ny * (nz / 2 + 1) + ctas - 1) / ctas),
        plane_elems((size_t)planes * fft_plane_elems(ny, nz)), list(list_capacity) {}
  __host__ __device__ size_t bytes(int nx, int ny, int nz) const {
    return 2 * sizeof(Real) * ((size_t)nx + ny + nz + 2 * plane_elems + 2 * (size_t)pencils * nx) +
           (sizeof(double) + 30 * sizeof(Real) + 4 * sizeof(int)) * (size_t)list +
           2 * sizeof(int) * (size_t)planes * ny * nz;
  }
};

template <class Real, int kTerms>
__global__ void __launch_bounds__(kClusterThreads) pme_cluster(const PmeArgs<Real> a, const PmeFft f,
                                                               int list_capacity) {
  using C2 = typename Cplx<Real>::T;
  extern __shared__ __align__(16) unsigned char fsm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int ctas = gridDim.x, rank = blockIdx.x;  // one cluster
  const int nx = a.nx, ny = a.ny, nz = a.nz, nzh = nz / 2 + 1, nyp = (ny + 1) / 2;
  const ClusterLayout<Real> L(nx, ny, nz, ctas, list_capacity);
  C2* twx = reinterpret_cast<C2*>(fsm);
  C2* twy = twx + nx;
  C2* twz = twy + ny;
  C2* A = twz + nz;
  C2* B = A + L.plane_elems;
  C2* XA = B + L.plane_elems;
  C2* XB = XA + (size_t)L.pencils * nx;
  double* l_q = reinterpret_cast<double*>(XB + (size_t)L.pencils * nx);  // the particle list:
  Real* l_w = reinterpret_cast<Real*>(l_q + L.list);          // [30][list] weights, then slopes
  int* l_base = reinterpret_cast<int*>(l_w + 30 * (size_t)L.list);  // [3][list]
  int* l_at = l_base + 3 * (size_t)L.list;
  int* c_hi = l_at + L.list;
  unsigned* c_lo = reinterpret_cast<unsigned*>(c_hi + (size_t)L.planes * ny * nz);
  const int x0 = rank * L.planes, np = max(0, min(L.planes, nx - x0));  // own planes
  load_twiddles(twx, f.tw[0], nx);
  load_twiddles(twy, f.tw[1], ny);
  load_twiddles(twz, f.tw[2], nz);
  for (int c = threadIdx.x; c < np * ny * nz; c += blockDim.x) {
    c_hi[c] = 0;
    c_lo[c] = 0u;
  }
  __syncthreads();
  // The particles whose stencils touch this CTA's planes (a quarter of them at 23 planes over 16
  // CTAs) are listed with their spline weights, kClusterThreads particles at a time: each thread
  // forms one stencil, and the work on those that count spreads evenly over every thread.  The
  // order of the list does not matter: the grid's and the forces' sums are fixed point.  A list
  // that holds every particle of this CTA is kept for the gather.
  __shared__ int s_n;
  auto weight = [&](int d, int k, int e) -> Real& { return l_w[(5 * d + k) * L.list + e]; };
  auto slope = [&](int d, int k, int e) -> Real& { return l_w[(15 + 5 * d + k) * L.list + e]; };
  bool whole = false;  // the list holds all of this CTA's particles
  auto for_each_list = [&](auto use) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    int lists = 0;
    for (int i0 = 0; i0 < a.n_atoms; i0 += kClusterThreads) {
      const int i = i0 + threadIdx.x;
      const double q = i < a.n_atoms ? a.charge[i] : 0.0;
      int base[3] = {0, 0, 0};
      Real frac[3] = {Real(0), Real(0), Real(0)};
      bool mine = q != 0.0 && stencil(a, i, base, frac);
      if (mine) {  // planes base .. base + 4, cyclic, against x0 .. x0 + np - 1
        int first = x0 - base[0];
        first += first < 0 ? nx : 0;  // distance from the base to the first own plane
        mine = np > 0 && (first < 5 || first + np > nx);
      }
      const unsigned m = __ballot_sync(0xffffffffu, mine);
      int at = 0;
      if (lane == 0 && m) at = atomicAdd(&s_n, __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
      if (mine) {
        l_at[at] = i;
        l_q[at] = q;
        for (int d = 0; d < 3; ++d) l_base[d * L.list + at] = base[d];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          Real w[5], dw[5];
          spline5(frac[d], w, dw);
#pragma unroll
          for (int k = 0; k < 5; ++k) {
            weight(d, k, at) = w[k];
            slope(d, k, at) = dw[k];
          }
        }
      }
      __syncthreads();
      const int n = s_n;
      __syncthreads();  // every thread has read the count before the next particles add to it
      const bool last = i0 + kClusterThreads >= a.n_atoms;
      if (last || n > L.list - kClusterThreads) {
        use(n);
        ++lists;
        __syncthreads();
        if (!last) {
          if (threadIdx.x == 0) s_n = 0;
          __syncthreads();
        }
      }
    }
    whole = lists == 1;
  };
  // own plane p of a particle with base plane b: the stencil plane it is, or >= 5
  auto stencil_plane = [&](int b, int p) {
    const int ix = x0 + p - b;
    return ix < 0 ? ix + nx : ix;
  };
  // spread (pme.rs:176-238): a thread takes one row in y of one own plane of a particle
  for_each_list([&](int n) {
    for (int t = threadIdx.x; t < 5 * np * n; t += blockDim.x) {
      const int e = t / (5 * np), r = t - e * 5 * np, p = r / 5, iy = r - 5 * p;
      const int ix = stencil_plane(l_base[e], p);
      if (ix >= 5) continue;
      int gy = l_base[L.list + e] + iy;
      gy -= gy >= ny ? ny : 0;
      const int bz = l_base[2 * L.list + e], row = (p * ny + gy) * nz;
      const Real qxy = (Real)l_q[e] * weight(0, ix, e) * weight(1, iy, e);
#pragma unroll
      for (int iz = 0; iz < 5; ++iz) {
        int gz = bz + iz;
        gz -= gz >= nz ? nz : 0;
        const Real v = qxy * weight(2, iz, e);
        int hi;
        unsigned lo;
        if constexpr (sizeof(Real) == 4) {  // v 2^40 to an integer, in 32-bit steps
          const float scaled = v * 1048576.f, whole_part = floorf(scaled);
          hi = (int)whole_part;
          lo = (unsigned)__float2int_rn((scaled - whole_part) * 1048576.f);
        } else {
          const long long f = to_fixed(v, Real(kGridScale));
          hi = (int)(f >> 20);
          lo = (unsigned)(f & 0xFFFFF);
        }
        atomicAdd(&c_hi[row + gz], hi);
        atomicAdd(&c_lo[row + gz], lo);
      }
    }
  });
  // rows y = 2 yp (real part) and 2 yp + 1 (imaginary part) as one complex row, z transform
  for (int i = threadIdx.x; i < np * nyp * nz; i += blockDim.x) {
    const int z = i % nz, r = i / nz, lp = r / nyp, yp = r - lp * nyp;
    const int c0 = (lp * ny + 2 * yp) * nz + z;
    C2 v;
    v.x = (Real)((double)((long long)c_hi[c0] * (1ll << 20) + (long long)c_lo[c0]) * kGridScaleInv);
    v.y = 0;
    if (2 * yp + 1 < ny) {
      const int c1 = c0 + nz;
      v.y = (Real)((double)((long long)c_hi[c1] * (1ll << 20) + (long long)c_lo[c1]) * kGridScaleInv);
    }
    A[i] = v;
  }
  __syncthreads();
  C2* r = stockham(A, B, twz, f, 2, nz, np * nyp);
  C2* o = r == A ? B : A;
  // split the two real rows' spectra into pencils along y: o[plane][kz][y] (planes_forward)
  for (int i = threadIdx.x; i < np * nzh * ny; i += blockDim.x) {
    const int y = i % ny, t = i / ny, lp = t / nzh, kz = t - lp * nzh, yp = y >> 1;
    const C2* row = r + (lp * nyp + yp) * nz;
    const C2 zk = row[kz], zm = row[kz == 0 ? 0 : nz - kz];
    C2 v;
    if ((y & 1) == 0) {
      v.x = (Real)0.5 * (zk.x + zm.x);
      v.y = (Real)0.5 * (zk.y - zm.y);
    } else {
      v.x = (Real)0.5 * (zk.y + zm.y);
      v.y = (Real)0.5 * (zm.x - zk.x);
    }
    o[i] = v;
  }
  __syncthreads();
  // the same buffer in every CTA: the swaps depend on the axes' stage counts alone
  C2* s = stockham(o, r, twy, f, 1, ny, np * nzh);
  cluster.sync();
  // x pass over this CTA's pencils q = kz ny + y
  const int q0 = rank * L.pencils, nq = max(0, min(L.pencils, nzh * ny - q0));
  for (int i = threadIdx.x; i < nq * nx; i += blockDim.x) {
    const int x = i / nq, q = i - x * nq, owner = x / L.planes, lp = x - owner * L.planes;
    XA[q * nx + x] = cluster.map_shared_rank(s, owner)[lp * nzh * ny + q0 + q];
  }
  __syncthreads();
  C2* xr = stockham(XA, XB, twx, f, 0, nx, nq);
  C2* xo = xr == XA ? XB : XA;
  double e = 0.0, vir[6] = {0, 0, 0, 0, 0, 0};
  for (int i = threadIdx.x; i < nq * nx; i += blockDim.x) {
    const int q = i / nx, x = i - q * nx, kz = (q0 + q) / ny, y = q0 + q - kz * ny;
    const long long at = ((long long)x * ny + y) * nzh + kz;
    const Real infl = __ldg(a.influence + at);
    C2 v = xr[i];
    if (kTerms && at != 0)
      mode_energy<kTerms>(a, x, y, kz, (double)v.x * v.x + (double)v.y * v.y, (double)infl, e, vir);
    v.x *= infl;
    v.y *= -infl;  // conjugated for the inverse transform
    xr[i] = v;
  }
  if (kTerms) commit_energy<kTerms>(a, e, vir);
  __syncthreads();
  C2* xs = stockham(xr, xo, twx, f, 0, nx, nq);
  // back to the owners, still conjugated: the inverse y transform starts from conj H.  Each
  // element was read, and is written, by this CTA alone
  for (int i = threadIdx.x; i < nq * nx; i += blockDim.x) {
    const int x = i / nq, q = i - x * nq, owner = x / L.planes, lp = x - owner * L.planes;
    cluster.map_shared_rank(s, owner)[lp * nzh * ny + q0 + q] = xs[q * nx + x];
  }
  cluster.sync();
  C2* h = stockham(s, s == A ? B : A, twy, f, 1, ny, np * nzh);
  C2* g = h == A ? B : A;
  // rows 2 yp and 2 yp + 1, Hermitian-completed along z, as one conjugated row (planes_inverse)
  for (int i = threadIdx.x; i < np * nyp * nz; i += blockDim.x) {
    const int k = i % nz, t = i / nz, lp = t / nyp, y0 = 2 * (t - lp * nyp);
    const bool low = k < nzh;
    const C2* col = h + ((size_t)lp * nzh + (low ? k : nz - k)) * ny + y0;
    C2 ca = col[0];
    if (!low) ca = conjg(ca);
    C2 cb;
    cb.x = cb.y = 0;
    if (y0 + 1 < ny) {
      cb = col[1];
      if (!low) cb = conjg(cb);
    }
    C2 v;
    v.x = ca.x + cb.y;
    v.y = ca.y - cb.x;
    g[i] = v;
  }
  __syncthreads();
  const C2* pot = stockham(g, h, twz, f, 2, nz, np * nyp);  // row 2 yp = Re, row 2 yp + 1 = -Im
  // gather (pme.rs:377-425): this CTA's planes' part of each listed particle's force, eight lanes
  // to a particle, five of them with a row in y each
  auto gather = [&](int n) {
    const int k = threadIdx.x & 7;
    for (int e0 = 0; e0 < n; e0 += kClusterThreads / 8) {
      const int e = e0 + (threadIdx.x >> 3);
      Real g0 = 0, g1 = 0, g2 = 0;
      if (e < n && k < 5) {
        int gy = l_base[L.list + e] + k;
        gy -= gy >= ny ? ny : 0;
        const int bx = l_base[e], bz = l_base[2 * L.list + e];
        for (int p = 0; p < np; ++p) {
          const int ix = stencil_plane(bx, p);
          if (ix >= 5) continue;
          const C2* row = pot + (p * nyp + (gy >> 1)) * nz;
          Real sum = 0, dsum = 0;
#pragma unroll
          for (int iz = 0; iz < 5; ++iz) {
            int gz = bz + iz;
            gz -= gz >= nz ? nz : 0;
            const C2 v = row[gz];
            const Real phi = (gy & 1) ? -v.y : v.x;
            sum += phi * weight(2, iz, e);
            dsum += phi * slope(2, iz, e);
          }
          g0 += slope(0, ix, e) * sum;
          g1 += weight(0, ix, e) * sum;
          g2 += weight(0, ix, e) * dsum;
        }
        g0 *= weight(1, k, e);
        g1 *= slope(1, k, e);
        g2 *= weight(1, k, e);
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) {
        g0 += __shfl_xor_sync(0xffffffffu, g0, o, 8);
        g1 += __shfl_xor_sync(0xffffffffu, g1, o, 8);
        g2 += __shfl_xor_sync(0xffffffffu, g2, o, 8);
      }
      if (e < n && k < 3) {  // one component per lane
        const double gd[3] = {(double)g0 * nx, (double)g1 * ny, (double)g2 * nz};
        const double fc =
            -l_q[e] * (gd[0] * a.recip[0][k] + gd[1] * a.recip[1][k] + gd[2] * a.recip[2][k]);
        add_fixed(a.force + (long long)k * a.n_atoms + l_at[e], to_fixed(fc, kForceScale));
      }
    }
  };
  if (whole)
    gather(s_n);
  else
    for_each_list(gather);
}

}  // namespace

template <class Real>
size_t pme_transform_smem(const PmeArgs<Real>& a, const PmeFft& f, int kernel) {
  using C2 = typename Cplx<Real>::T;
  if (kernel == 1) return sizeof(C2) * (size_t)a.nx * (1 + 2 * f.pencils_x);
  return sizeof(C2) * ((size_t)a.ny + a.nz + 2 * (size_t)fft_plane_elems(a.ny, a.nz));
}

template <class Real>
void launch_pme_transform(const PmeArgs<Real>& a, const PmeFft& f, int terms, cudaStream_t s) {
  const size_t sp = pme_transform_smem(a, f, 0), sx = pme_transform_smem(a, f, 1);
  const int nzh = a.nz / 2 + 1, nkb = ceil_div(nzh, f.pencils_x);
  planes_forward<Real><<<a.nx, f.threads[0], sp, s>>>(a, f);
  if (terms == kTermsVirial)
    x_convolve<Real, kTermsVirial><<<a.ny * nkb, f.threads[1], sx, s>>>(a, f);
  else if (terms == kTermsEnergy)
    x_convolve<Real, kTermsEnergy><<<a.ny * nkb, f.threads[1], sx, s>>>(a, f);
  else
    x_convolve<Real, kTermsNone><<<a.ny * nkb, f.threads[1], sx, s>>>(a, f);
  planes_inverse<Real><<<a.nx, f.threads[2], sp, s>>>(a, f);
}

template <class Real>
void prepare_pme_transform(const PmeArgs<Real>& a, const PmeFft& f) {
  const int sp = (int)pme_transform_smem(a, f, 0), sx = (int)pme_transform_smem(a, f, 1);
  cudaFuncSetAttribute((const void*)planes_forward<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp);
  cudaFuncSetAttribute((const void*)planes_inverse<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize, sp);
  cudaFuncSetAttribute((const void*)x_convolve<Real, kTermsVirial>, cudaFuncAttributeMaxDynamicSharedMemorySize, sx);
  cudaFuncSetAttribute((const void*)x_convolve<Real, kTermsEnergy>, cudaFuncAttributeMaxDynamicSharedMemorySize, sx);
  cudaFuncSetAttribute((const void*)x_convolve<Real, kTermsNone>, cudaFuncAttributeMaxDynamicSharedMemorySize, sx);
}

// Capacity of the cluster form's particle lists: two batches, or one where shared memory is short.
constexpr size_t kClusterSmem = 200 * 1024;
template <class Real>
int cluster_list(const PmeArgs<Real>& a, int ctas) {
  const ClusterLayout<Real> two(a.nx, a.ny, a.nz, ctas, 2 * kClusterThreads);
  return two.bytes(a.nx, a.ny, a.nz) <= kClusterSmem ? 2 * kClusterThreads : kClusterThreads;
}

// The cluster form's launch: `ctas` CTAs of one cluster.
template <class Real, int kTerms>
cudaLaunchConfig_t cluster_config(const PmeArgs<Real>& a, int ctas, cudaLaunchAttribute* attr,
                                  cudaStream_t s) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes =
      ClusterLayout<Real>(a.nx, a.ny, a.nz, ctas, cluster_list(a, ctas)).bytes(a.nx, a.ny, a.nz);
  cfg.stream = s;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = ctas;
  attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

template <class Real, int kTerms>
bool prepare_cluster(const PmeArgs<Real>& a, int ctas) {
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cluster_config<Real, kTerms>(a, ctas, &attr, nullptr);
  if (cfg.dynamicSmemBytes > kClusterSmem) return false;
  auto* fn = pme_cluster<Real, kTerms>;
  if (cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)cfg.dynamicSmemBytes) != cudaSuccess ||
      (ctas > 8 && cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeNonPortableClusterSizeAllowed,
                                        1) != cudaSuccess)) {
    cudaGetLastError();
    return false;
  }
  int clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) != cudaSuccess) cudaGetLastError();
  return clusters > 0;
}

template <class Real>
int pme_cluster_ctas(const PmeArgs<Real>& a) {
  if (a.n_atoms > kClusterAtoms) return 0;
  for (int ctas : {16, 8})
    if (prepare_cluster<Real, kTermsNone>(a, ctas) && prepare_cluster<Real, kTermsEnergy>(a, ctas) &&
        prepare_cluster<Real, kTermsVirial>(a, ctas))
      return ctas;
  return 0;
}

template <class Real, int kTerms>
void launch_cluster(const PmeArgs<Real>& a, const PmeFft& f, int ctas, cudaStream_t s) {
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cluster_config<Real, kTerms>(a, ctas, &attr, s);
  cudaLaunchKernelEx(&cfg, pme_cluster<Real, kTerms>, a, f, cluster_list(a, ctas));
}

template <class Real>
void launch_pme_cluster(const PmeArgs<Real>& a, const PmeFft& f, int ctas, int terms,
                        cudaStream_t s) {
  if (terms == kTermsVirial)
    launch_cluster<Real, kTermsVirial>(a, f, ctas, s);
  else if (terms == kTermsEnergy)
    launch_cluster<Real, kTermsEnergy>(a, f, ctas, s);
  else
    launch_cluster<Real, kTermsNone>(a, f, ctas, s);
}

template int pme_cluster_ctas<float>(const PmeArgs<float>&);
template int pme_cluster_ctas<double>(const PmeArgs<double>&);
template void launch_pme_cluster<float>(const PmeArgs<float>&, const PmeFft&, int, int, cudaStream_t);
template void launch_pme_cluster<double>(const PmeArgs<double>&, const PmeFft&, int, int, cudaStream_t);
template size_t pme_transform_smem<float>(const PmeArgs<float>&, const PmeFft&, int);
template size_t pme_transform_smem<double>(const PmeArgs<double>&, const PmeFft&, int);
template void launch_pme_transform<float>(const PmeArgs<float>&, const PmeFft&, int, cudaStream_t);
template void launch_pme_transform<double>(const PmeArgs<double>&, const PmeFft&, int, cudaStream_t);
template void prepare_pme_transform<float>(const PmeArgs<float>&, const PmeFft&);
template void prepare_pme_transform<double>(const PmeArgs<double>&, const PmeFft&);

namespace {
// pme.rs:332-350: the influence function on the half spectrum, averaged over each mode and its
// conjugate partner, zero at k = 0 (one thread per half-grid point, f64).
template <class Real>
__global__ void influence_kernel(Real* out, const double* moduli, int nx, int ny, int nz,
                                 PmeRecip r, double alpha, double volume) {
  const int nzh = nz / 2 + 1;
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= (long long)nx * ny * nzh) return;
  const int z = (int)(i % nzh), y = (int)((i / nzh) % ny), x = (int)(i / ((long long)nzh * ny));
  if (i == 0) {
    out[0] = Real(0);
    return;
  }
  const double pa = kPiD * kPiD / (alpha * alpha);
  auto g = [&](int gx, int gy, int gz) {
    const double m[3] = {freq(gx, nx), freq(gy, ny), freq(gz, nz)};
    double k2 = 0.0;
    for (int c = 0; c < 3; ++c) {
      const double kc = m[0] * r.m[0][c] + m[1] * r.m[1][c] + m[2] * r.m[2][c];
      k2 += kc * kc;
    }
    return kOne4PiEps0 * exp(-pa * k2) /
           (kPiD * volume * k2 * moduli[gx] * moduli[nx + gy] * moduli[nx + ny + gz]);
  };
  out[i] = (Real)(0.5 * (g(x, y, z) + g((nx - x) % nx, (ny - y) % ny, (nz - z) % nz)));
}
}  // namespace

template <class Real>
void launch_pme_influence(Real* out, const double* moduli, int nx, int ny, int nz,
                          const PmeRecip& recip, double alpha, double volume, cudaStream_t s) {
  const long long n = (long long)nx * ny * (nz / 2 + 1);
  influence_kernel<Real><<<(int)((n + 255) / 256), 256, 0, s>>>(out, moduli, nx, ny, nz, recip,
                                                                alpha, volume);
}
template void launch_pme_influence<float>(float*, const double*, int, int, int, const PmeRecip&,
                                          double, double, cudaStream_t);
template void launch_pme_influence<double>(double*, const double*, int, int, int, const PmeRecip&,
                                           double, double, cudaStream_t);

template <class Real>
void launch_pme_spread(const PmeArgs<Real>& a, cudaStream_t s) {
  if (a.order) {  // sorted slots: spatially compact CTAs
    spread_staged_kernel<Real><<<ceil_div(a.n_order, kSpreadAtoms), 2 * kSpreadAtoms, 0, s>>>(a);
  } else {
    spread_kernel<Real><<<ceil_div(a.n_order, 128), 128, 0, s>>>(a);
  }
}
template <class Real>
void launch_pme_convert(const PmeArgs<Real>& a, cudaStream_t s) {
  const long long total = (long long)a.nx * a.ny * a.nz;
  convert_kernel<Real><<<(int)std::min<long long>((total + 255) / 256, 148LL * 16), 256, 0, s>>>(a);
}
template <class Real>
void launch_pme_convolve(const PmeArgs<Real>& a, int terms, cudaStream_t s) {
  const long long total = (long long)a.nx * a.ny * (a.nz / 2 + 1);
  const int grid = (int)std::min<long long>((total + 255) / 256, 148LL * 16);
  if (terms == kTermsVirial)
    convolve_kernel<Real, kTermsVirial><<<grid, 256, 0, s>>>(a);
  else if (terms == kTermsEnergy)
    convolve_kernel<Real, kTermsEnergy><<<grid, 256, 0, s>>>(a);
  else
    convolve_kernel<Real, kTermsNone><<<grid, 256, 0, s>>>(a);
}
template <class Real>
void launch_pme_gather(const PmeArgs<Real>& a, cudaStream_t s) {
  gather_kernel<Real><<<ceil_div((long long)a.n_order * 8, 128), 128, 0, s>>>(a);
}

template void launch_pme_spread<float>(const PmeArgs<float>&, cudaStream_t);
template void launch_pme_spread<double>(const PmeArgs<double>&, cudaStream_t);
template void launch_pme_convert<float>(const PmeArgs<float>&, cudaStream_t);
template void launch_pme_convert<double>(const PmeArgs<double>&, cudaStream_t);
template void launch_pme_convolve<float>(const PmeArgs<float>&, int, cudaStream_t);
template void launch_pme_convolve<double>(const PmeArgs<double>&, int, cudaStream_t);
template void launch_pme_gather<float>(const PmeArgs<float>&, cudaStream_t);
template void launch_pme_gather<double>(const PmeArgs<double>&, cudaStream_t);

// ---- brick-owned gathering --------------------------------------------------------------
// For large grids in rectangular boxes.  A first kernel stores every slot's stencil (base point,
// fractions, charge).  Then one CTA per brick of kBrickEdge^3 grid points reads the brick and
// its 4-point halo of the potential grid into shared memory once, collects its candidates from
// the per-rebuild slot ranges of the x-y columns in reach (one 16-byte stencil load each), and
// takes those whose stencil starts inside the brick, so every particle is gathered by one CTA
// from shared memory instead of by eight lanes from L2.  Each atom's stencil planes are summed
// in the order of the eight-lane kernel, so both forms give the same forces.  (A brick-owned
// spread, storing each brick's sums once, measured slower than the atomic spread on the 196^3
// grid: its shared-memory sums cost more than the global atomics they replace.)
namespace {

constexpr int kBrickThreads = 256;
constexpr int kBrickHalo = (kBrickEdge + 4) * (kBrickEdge + 4) * (kBrickEdge + 4);
constexpr int kBrickOwnChunk = 2048;  // candidates tested before their owners are gathered
static_assert(kBrickMaxRanges <= kBrickThreads, "one range per thread when collecting");

// first slot k in [s0, s0 + n) of a z-sorted column with zkey >= z (s0 + n if none)
__device__ int column_lower(const NlistArgs& a, int s0, int n, float z) {
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (a.zkey[a.sorted_atom[s0 + mid]] < z)
      lo = mid + 1;
    else
      hi = mid;
  }
  return s0 + lo;
}

// One thread per (column, z layer of bricks): the slots of the column's atoms whose wrapped
// rebuild z lies within the layer's reach, as one range or two (the reach wraps the box).
__global__ void brick_ranges_kernel(const NlistArgs a, const PmeBricks b) {
  if (*a.rebuild == 0) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n_cols * b.nb[2]) return;
  const int c = i % a.n_cols, bz = i / a.n_cols;
  const int s0 = a.col_start[c];
  const int n = min(a.col_size[c], a.col_max);
  const double L = b.len[2];
  const double z0 = bz * kBrickEdge * b.cell[2] - b.below[2];
  const double z1 = min((bz + 1) * kBrickEdge, b.grid[2]) * b.cell[2] + b.above;
  int2 r0 = make_int2(s0, s0), r1 = make_int2(s0, s0);
  if (z1 - z0 >= L) {
    r0.y = s0 + n;
  } else if (z0 < 0.0) {
    r0 = make_int2(column_lower(a, s0, n, (float)(z0 + L)), s0 + n);
    r1 = make_int2(s0, column_lower(a, s0, n, (float)z1));
  } else if (z1 > L) {
    r0 = make_int2(column_lower(a, s0, n, (float)z0), s0 + n);
    r1 = make_int2(s0, column_lower(a, s0, n, (float)(z1 - L)));
  } else {
    r0 = make_int2(column_lower(a, s0, n, (float)z0), column_lower(a, s0, n, (float)z1));
  }
  b.ranges[2 * i] = r0;
  b.ranges[2 * i + 1] = r1;
}

// first grid point and extent of brick `id` along each axis
__device__ __forceinline__ void brick_box(const PmeBricks& b, int id, int b0[3], int e[3],
                                          int bi[3]) {
  bi[0] = id % b.nb[0];
  bi[1] = (id / b.nb[0]) % b.nb[1];
  bi[2] = id / (b.nb[0] * b.nb[1]);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    b0[d] = bi[d] * kBrickEdge;
    e[d] = min(kBrickEdge, b.grid[d] - b0[d]);
  }
}

// columns along axis d (0: x, 1: y) whose rebuild positions can reach brick index bd
__device__ __forceinline__ void column_span(const PmeBricks& b, int d, int bd, int& c0, int& nc) {
  const int ncol = b.n_col[d];
  const double w = b.len[d] / ncol;
  const double lo = bd * kBrickEdge * b.cell[d] - b.below[d];
  const double hi = min((bd + 1) * kBrickEdge, b.grid[d]) * b.cell[d] + b.above;
  c0 = (int)floor(lo / w);
  nc = (int)floor(hi / w) - c0 + 1;
  if (nc >= ncol) {
    c0 = 0;
    nc = ncol;
  }
}

// The brick's candidate slot ranges into s_rng, their exclusive prefix into s_pre; returns the
// number of ranges (the candidate count is s_pre[ranges]).  Block-wide, with barriers.
__device__ int brick_candidates(const PmeBricks& b, const NlistArgs& nl, const int bi[3],
                                int2* s_rng, int* s_pre, int* s_warp) {
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  int cx0, ncx, cy0, ncy;
  column_span(b, 0, bi[0], cx0, ncx);
  column_span(b, 1, bi[1], cy0, ncy);
  const int nr = min(2 * ncx * ncy, kBrickMaxRanges);  // the host keeps 2 ncx ncy within
  int len = 0;
  if (t < nr) {
    const int k = t >> 1, piece = t & 1;
    int cx = (cx0 + k % ncx) % b.n_col[0];
    int cy = (cy0 + k / ncx) % b.n_col[1];
    cx += cx < 0 ? b.n_col[0] : 0;
    cy += cy < 0 ? b.n_col[1] : 0;
    const int col = cy * b.n_col[0] + cx;
    const int2 r = b.ranges[2 * ((size_t)bi[2] * nl.n_cols + col) + piece];
    s_rng[t] = r;
    len = max(r.y - r.x, 0);
  }
  int incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) s_warp[w] = incl;
  __syncthreads();
  if (w == 0) {
    int v = lane < kBrickThreads / 32 ? s_warp[lane] : 0, x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane < kBrickThreads / 32) s_warp[lane] = x - v;  // exclusive warp offsets
  }
  __syncthreads();
  const int excl = incl - len + s_warp[w];
  if (t < nr) s_pre[t] = excl;
  if (t == nr - 1) s_pre[nr] = excl + len;
  __syncthreads();
  return nr;
}

// slot of candidate i: the last range whose prefix does not exceed i holds it
__device__ __forceinline__ int candidate_slot(const int2* s_rng, const int* s_pre, int nr, int i) {
  int lo = 0, hi = nr - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (s_pre[mid] <= i)
      lo = mid;
    else
      hi = mid - 1;
  }
  return s_rng[lo].x + (i - s_pre[lo]);
}

template <class Real>
struct Real4Of;
template <>
struct Real4Of<float> {
  using T = float4;
};
template <>
struct Real4Of<double> {
  using T = double4;
};

// This step's stencil of every sorted slot (the spread and the gather of the brick form read it
// once per candidate instead of recomputing it from the position): base point per axis and the
// fractions, as `stencil` gives them, and the charge as Real.
template <class Real>
__global__ void brick_stencils_kernel(const PmeArgs<Real> a, const PmeBricks b, const NlistArgs nl) {
  using R4 = typename Real4Of<Real>::T;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= b.n_slots) return;
  const int atom = nl.sorted_atom[s];
  const double qd = atom >= 0 ? a.charge[atom] : 0.0;
  int base[3] = {0, 0, 0};
  Real frac[3] = {Real(0), Real(0), Real(0)};
  const bool ok = qd != 0.0 && stencil(a, atom, base, frac);
  b.base[s] = make_int4(base[0], base[1], base[2], ok ? 1 : 0);
  R4 f;
  f.x = frac[0];
  f.y = frac[1];
  f.z = frac[2];
  f.w = (Real)qd;
  reinterpret_cast<R4*>(b.frac)[s] = f;
}

template <class Real>
__global__ void __launch_bounds__(kBrickThreads) gather_bricks_kernel(const PmeArgs<Real> a,
                                                                      const PmeBricks b,
                                                                      const NlistArgs nl) {
  using R4 = typename Real4Of<Real>::T;
  extern __shared__ __align__(16) unsigned char brick_smem[];
  Real* phi = reinterpret_cast<Real*>(brick_smem);  // [(e0 + 4)(e1 + 4)(e2 + 4)]
  __shared__ int2 s_rng[kBrickMaxRanges];
  __shared__ int s_pre[kBrickMaxRanges + 1];
  __shared__ int s_warp[kBrickThreads / 32];
  __shared__ int s_own[kBrickOwnChunk];
  __shared__ int s_nown;
  int b0[3], e[3], bi[3];
  brick_box(b, blockIdx.x, b0, e, bi);
  const int h1 = e[1] + 4, h2 = e[2] + 4, nh = (e[0] + 4) * h1 * h2;
  for (int c = threadIdx.x; c < nh; c += kBrickThreads) {
    const int hz = c % h2, hy = (c / h2) % h1, hx = c / (h1 * h2);
    int gx = b0[0] + hx, gy = b0[1] + hy, gz = b0[2] + hz;
    gx -= gx >= a.nx ? a.nx : 0;
    gy -= gy >= a.ny ? a.ny : 0;
    gz -= gz >= a.nz ? a.nz : 0;
    phi[c] = a.grid_real[((long long)gx * a.ny + gy) * a.nz + gz];
  }
  const int nr = brick_candidates(b, nl, bi, s_rng, s_pre, s_warp);  // barriers cover phi
  const int n_cand = s_pre[nr];
  // The candidates are tested in chunks; the owners (stencil starting in this brick, about a
  // third) are listed in shared memory and then gathered one per thread, so that the 125-point
  // sums run on full warps.  The order of the list does not matter: each particle's force is
  // its own sum, added in fixed point.
  for (int i0 = 0; i0 < n_cand; i0 += kBrickOwnChunk) {
    if (threadIdx.x == 0) s_nown = 0;
    __syncthreads();
    const int i1 = min(i0 + kBrickOwnChunk, n_cand);
    for (int i = i0 + threadIdx.x; i < i1; i += kBrickThreads) {
      const int slot = candidate_slot(s_rng, s_pre, nr, i);
      const int4 sb = b.base[slot];
      const bool own = sb.w && (unsigned)(sb.x - b0[0]) < (unsigned)e[0] &&
                       (unsigned)(sb.y - b0[1]) < (unsigned)e[1] &&
                       (unsigned)(sb.z - b0[2]) < (unsigned)e[2];
      const unsigned m = __ballot_sync(__activemask(), own);
      if (own) {
        const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
        int at = 0;
        if (lane == leader) at = atomicAdd(&s_nown, __popc(m));
        at = __shfl_sync(m, at, leader) + __popc(m & ((1u << lane) - 1u));
        s_own[at] = slot;
      }
    }
    __syncthreads();
    const int n_own = s_nown;
    for (int o = threadIdx.x; o < n_own; o += kBrickThreads) {
    const int slot = s_own[o];
    const int4 sb = b.base[slot];
    const int lx = sb.x - b0[0], ly = sb.y - b0[1], lz = sb.z - b0[2];
    const R4 sf = reinterpret_cast<const R4*>(b.frac)[slot];
    const int atom = nl.sorted_atom[slot];
    const double qd = a.charge[atom];
    Real w[3][5], dw[3][5];
    spline5(sf.x, w[0], dw[0]);
    spline5(sf.y, w[1], dw[1]);
    spline5(sf.z, w[2], dw[2]);
    Real p0[5], p1[5], p2[5];  // stencil plane ix: the sums of lane ix of the eight-lane kernel
#pragma unroll
    for (int ix = 0; ix < 5; ++ix) {
      Real g0 = 0, g1 = 0, g2 = 0;
      const Real wx = w[0][ix], dwx = dw[0][ix];
      for (int iy = 0; iy < 5; ++iy) {
        const Real* row = phi + ((lx + ix) * h1 + (ly + iy)) * h2 + lz;
        const Real wxy = wx * w[1][iy];
        const Real dxy = dwx * w[1][iy];
        const Real xdy = wx * dw[1][iy];
#pragma unroll
        for (int iz = 0; iz < 5; ++iz) {
          const Real ph = row[iz];
          g0 += ph * dxy * w[2][iz];
          g1 += ph * xdy * w[2][iz];
          g2 += ph * wxy * dw[2][iz];
        }
      }
      p0[ix] = g0;
      p1[ix] = g1;
      p2[ix] = g2;
    }
    // the eight-lane kernel's xor tree (lanes 5-7 hold zeros)
    const Real g0 = ((p0[0] + p0[4]) + p0[2]) + (p0[1] + p0[3]);
    const Real g1 = ((p1[0] + p1[4]) + p1[2]) + (p1[1] + p1[3]);
    const Real g2 = ((p2[0] + p2[4]) + p2[2]) + (p2[1] + p2[3]);
    const double gd[3] = {(double)g0 * a.nx, (double)g1 * a.ny, (double)g2 * a.nz};
    for (int c = 0; c < 3; ++c) {
      const double f = -qd * (gd[0] * a.recip[0][c] + gd[1] * a.recip[1][c] + gd[2] * a.recip[2][c]);
      add_fixed(a.force + (long long)c * a.n_atoms + atom, to_fixed(f, kForceScale));
    }
    }
    __syncthreads();  // the list is refilled by the next chunk
  }
}

}  // namespace

void launch_pme_brick_ranges(const NlistArgs& a, const PmeBricks& b, cudaStream_t s) {
  const int n = a.n_cols * b.nb[2];
  brick_ranges_kernel<<<ceil_div(n, 128), 128, 0, s>>>(a, b);
}

template <class Real>
void launch_pme_brick_stencils(const PmeArgs<Real>& a, const PmeBricks& b, const NlistArgs& nl,
                               cudaStream_t s) {
  brick_stencils_kernel<Real><<<ceil_div(b.n_slots, 256), 256, 0, s>>>(a, b, nl);
}
template void launch_pme_brick_stencils<float>(const PmeArgs<float>&, const PmeBricks&,
                                               const NlistArgs&, cudaStream_t);
template void launch_pme_brick_stencils<double>(const PmeArgs<double>&, const PmeBricks&,
                                                const NlistArgs&, cudaStream_t);

template <class Real>
void launch_pme_gather_bricks(const PmeArgs<Real>& a, const PmeBricks& b, const NlistArgs& nl,
                              cudaStream_t s) {
  const int bytes = (int)(sizeof(Real) * kBrickHalo);  // the FP64 halo exceeds 48 KB with the rest
  cudaFuncSetAttribute(gather_bricks_kernel<Real>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       bytes);
  gather_bricks_kernel<Real><<<b.nb[0] * b.nb[1] * b.nb[2], kBrickThreads, bytes, s>>>(a, b, nl);
}

template void launch_pme_gather_bricks<float>(const PmeArgs<float>&, const PmeBricks&,
                                              const NlistArgs&, cudaStream_t);
template void launch_pme_gather_bricks<double>(const PmeArgs<double>&, const PmeBricks&,
                                               const NlistArgs&, cudaStream_t);

}  // namespace ommb200
