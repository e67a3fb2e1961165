// Flow control of the channel (auxiliaryRoutines.f90:336-540): the volume
// sums behind setPressGrad (the mean density at the ux faces) and
// computeFlowRate (the ux flux), and setFlowRate's uniform shift of ux.
// A sum runs over the ux faces i = 0..nx-1, j = 1..ny, k = 1..nz with the
// staggered volume Vsx(i,j,k) = dxc(i+1)*dyf(j)*dzf(k) (grid.f90:812-838):
// one warp per (j, k) row into a partial, then one block adds the partials
// in a fixed order, so a sum is the same on every call (its order differs
// from the reference's sequential loop: agreement to rounding).
#include <cuda_runtime.h>

#include "tbfp_kernels.cuh"

namespace tbfp {

namespace {

constexpr int kRT = 128;

constexpr int kRW = 8;  // rows per block, one per warp

// A warp adds one row, four loads in flight per lane, and folds it by shuffles
// (0.114 ms on 512x384x256 with a block of 128 threads and a shared-memory tree
// per row; now 0.084, 0.061 at the copy bandwidth).
template <int MODE>  // 0: 0.5*(rho(i+1)+rho(i)), 1: ux(i)
__global__ void __launch_bounds__(32 * kRW) k_face_sum_rows(const double *__restrict__ f, Lay L,
                                                            const double *__restrict__ dxc,
                                                            const double *__restrict__ dyf,
                                                            const double *__restrict__ dzf, int nx, int ny, int nz,
                                                            double *__restrict__ part) {
  const int lane = threadIdx.x & 31;
  const long row = (long)blockIdx.x * kRW + (threadIdx.x >> 5);
  if (row >= (long)ny * nz) return;
  const int j = (int)(row % ny) + 1, k = (int)(row / ny) + 1;
  const double dy = dyf[j - 1], dz = dzf[k - 1];
  const double *r = f + at(L, 0, j, k);
  double s = 0.0;
#pragma unroll 4
  for (int i = lane; i < nx; i += 32) {
    const double x = MODE == 0 ? 0.5 * (r[i + 1] + r[i]) : r[i];
    s += x * (dxc[i] * dy * dz);  // dxc(i+1)*dyf(j)*dzf(k)
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) part[row] = s;
}

__global__ void __launch_bounds__(1024) k_sum_partials(const double *__restrict__ part, long n,
                                                       double *__restrict__ out) {
  double s = 0.0;
  for (long e = threadIdx.x; e < n; e += 1024) s += part[e];
  __shared__ double red[1024];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = 512; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

// setFlowRate: ux(0:nx, 1:ny, 1:nz) += uf
__global__ void __launch_bounds__(kRT) k_add_ux(double *__restrict__ ux, Lay L, int nx, double uf) {
  const int i = blockIdx.x * kRT + threadIdx.x, j = blockIdx.y + 1, k = blockIdx.z + 1;
  if (i > nx) return;
  const long o = at(L, i, j, k);
  ux[o] = ux[o] + uf;
}

}  // namespace

void launch_face_sum(int mode, const double *f, Lay L, const double *dxc, const double *dyf, const double *dzf, int nx,
                     int ny, int nz, double *part, double *out, cudaStream_t st) {
  const unsigned grid = (unsigned)(((long)ny * nz + kRW - 1) / kRW);
  if (mode == 0) k_face_sum_rows<0><<<grid, 32 * kRW, 0, st>>>(f, L, dxc, dyf, dzf, nx, ny, nz, part);
  else k_face_sum_rows<1><<<grid, 32 * kRW, 0, st>>>(f, L, dxc, dyf, dzf, nx, ny, nz, part);
  k_sum_partials<<<1, 1024, 0, st>>>(part, (long)ny * nz, out);
}

void launch_add_ux(double *ux, Lay L, int nx, int ny, int nz, double uf, cudaStream_t st) {
  k_add_ux<<<dim3((nx + 1 + kRT - 1) / kRT, ny, nz), kRT, 0, st>>>(ux, L, nx, uf);
}

}  // namespace tbfp
