// What getState returns, computed on the device in the layout the caller receives: forces as
// f64 triples (the fixed-point sums are three arrays of n) and the kinetic energy.  Both are
// bound by the launch at the sizes they run at (3.2 and 3.9 us at 52,713 particles); they replace
// host loops over the copied arrays and, when the velocities are not asked for, their copy: with
// the small results read back in one wait, new positions in, forces and energy out take 832 us at
// 52,713 particles against 1,428.
#include "kernels.h"

namespace ommb200 {
namespace {

__global__ void __launch_bounds__(256) state_forces_kernel(int n, const long long* force,
                                                           double* out) {
  // consecutive threads write consecutive doubles; the three source arrays are read in runs
  const long long t = blockIdx.x * 256ll + threadIdx.x;
  if (t >= 3ll * n) return;
  const int i = (int)(t / 3), c = (int)(t - 3ll * i);
  out[t] = (double)force[(long long)c * n + i] * kForceScaleInv;
}

__global__ void __launch_bounds__(512) kinetic_energy_kernel(int n, const double* mass,
                                                             const double* vel, double* parts) {
  __shared__ double s_sum[16];
  double ke = 0.0;
  for (int i = blockIdx.x * 512 + threadIdx.x; i < n; i += kKineticParts * 512) {
    const double x = vel[3ll * i], y = vel[3ll * i + 1], z = vel[3ll * i + 2];
    ke += mass[i] * (x * x + y * y + z * z);
  }
  for (int o = 16; o > 0; o >>= 1) ke += __shfl_xor_sync(0xffffffffu, ke, o);
  if ((threadIdx.x & 31) == 0) s_sum[threadIdx.x >> 5] = ke;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < 16; ++w) s += s_sum[w];
    parts[blockIdx.x] = s;
  }
}

}  // namespace

void launch_state_forces(int n, const long long* force, double* out, cudaStream_t s) {
  state_forces_kernel<<<ceil_div(3ll * n, 256), 256, 0, s>>>(n, force, out);
}

void launch_kinetic_energy(int n, const double* mass, const double* vel, double* parts,
                           cudaStream_t s) {
  kinetic_energy_kernel<<<kKineticParts, 512, 0, s>>>(n, mass, vel, parts);
}

}  // namespace ommb200
