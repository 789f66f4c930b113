// fsl_inc.cu -- the incompressible fluctuating fluid (FSL_SCHEME_INCOMPRESSIBLE).
//
// The solver of keyword incompressible (src/runSchemeIncompressible.cu:
// 20-155), FP64 as the reference: staggered velocities u (Rep::v64), a
// Crank-Nicolson viscous term and a midpoint advection in two substeps that
// share one noise draw, each substep a W build in real space, a forward FFT,
// the shifted Crank-Nicolson solve with the divergence-free projection per
// mode, and an inverse FFT.  The prediction u^{n+1/2} = (v + u^n) / 2 of the
// first substep (src/realToComplex.cu:108-119), written by the inverse
// transform, lives in the 8-byte spread buffer (Rep::grid, unused by this
// scheme).  The transforms and the solve are those of fsl_fft_g.cu.
#include "fsl_internal.cuh"

namespace fsl {

namespace {

unsigned blocks_for(long work, int tb) { return (unsigned)((work + tb - 1) / tb); }

__device__ __forceinline__ int wrapi(int j, int m) { return j < 0 ? j + m : (j >= m ? j - m : j); }

// W = u + dt/2 (eta/rho) L u - (dt/4) A(a) + div(Sigma) per cell, the
// advection A of field a (u, or the prediction in the second substep),
// src/kernelConstructW.cu:32-265 and 266-521; the random stress is the
// traceless symmetric tensor with layout XX, XY, XZ, YY, YZ, ZZ.
template <bool ONE>
__global__ void k_inc_w(FSL_KARGS, int second) {
  FSL_REP_AT(blockIdx.y);
  const int mx = P.mx, my = P.my, mz = P.mz, nc = P.nc;
  const double* ux = R.v64;
  const double* uy = R.v64 + nc;
  const double* uz = R.v64 + 2 * (size_t)nc;
  const double* a = second ? reinterpret_cast<const double*>(R.grid) : R.v64;
  const double* ax = a;
  const double* ay = a + nc;
  const double* az = a + 2 * (size_t)nc;
  const double* Rn = R.noise64;
  const double idx = P.invdx, idy = P.invdy, idz = P.invdz, dt = P.dt;
  const double nu = P.eta / P.rho, f1 = P.fact1, f4 = P.fact4;
  const size_t n = (size_t)nc;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nc; i += gridDim.x * blockDim.x) {
    const int x = i % mx, y = (i / mx) % my, z = i / (mx * my);
    auto at = [&](int dx, int dy, int dz) {
      return wrapi(x + dx, mx) + mx * (wrapi(y + dy, my) + my * wrapi(z + dz, mz));
    };
    const int v0 = at(0, 0, -1), v1 = at(0, -1, 0), v2 = at(-1, 0, 0), v3 = at(1, 0, 0),
              v4 = at(0, 1, 0), v5 = at(0, 0, 1);
    const int pxmy = at(1, -1, 0), pxmz = at(1, 0, -1), mxpy = at(-1, 1, 0), mxpz = at(-1, 0, 1),
              pymz = at(0, 1, -1), mypz = at(0, -1, 1);
    double wx = idx * idx * (ux[v3] - 2 * ux[i] + ux[v2]);
    wx += idy * idy * (ux[v4] - 2 * ux[i] + ux[v1]);
    wx += idz * idz * (ux[v5] - 2 * ux[i] + ux[v0]);
    wx = 0.5 * dt * nu * wx;
    double wy = idx * idx * (uy[v3] - 2 * uy[i] + uy[v2]);
    wy += idy * idy * (uy[v4] - 2 * uy[i] + uy[v1]);
    wy += idz * idz * (uy[v5] - 2 * uy[i] + uy[v0]);
    wy = 0.5 * dt * nu * wy;
    double wz = idx * idx * (uz[v3] - 2 * uz[i] + uz[v2]);
    wz += idy * idy * (uz[v4] - 2 * uz[i] + uz[v1]);
    wz += idz * idz * (uz[v5] - 2 * uz[i] + uz[v0]);
    wz = 0.5 * dt * nu * wz;
    wx += ux[i];
    wy += uy[i];
    wz += uz[i];
    double advX = idx * ((ax[v3] + ax[i]) * (ax[v3] + ax[i]) - (ax[i] + ax[v2]) * (ax[i] + ax[v2]));
    advX += idy * ((ax[v4] + ax[i]) * (ay[v3] + ay[i]) - (ax[i] + ax[v1]) * (ay[pxmy] + ay[v1]));
    advX += idz * ((ax[v5] + ax[i]) * (az[v3] + az[i]) - (ax[i] + ax[v0]) * (az[pxmz] + az[v0]));
    advX = 0.25 * dt * advX;
    double advY = idx * ((ay[v3] + ay[i]) * (ax[v4] + ax[i]) - (ay[i] + ay[v2]) * (ax[mxpy] + ax[v2]));
    advY += idy * ((ay[v4] + ay[i]) * (ay[v4] + ay[i]) - (ay[i] + ay[v1]) * (ay[i] + ay[v1]));
    advY += idz * ((ay[v5] + ay[i]) * (az[v4] + az[i]) - (ay[i] + ay[v0]) * (az[pymz] + az[v0]));
    advY = 0.25 * dt * advY;
    double advZ = idx * ((az[v3] + az[i]) * (ax[v5] + ax[i]) - (az[i] + az[v2]) * (ax[mxpz] + ax[v2]));
    advZ += idy * ((az[v4] + az[i]) * (ay[v5] + ay[i]) - (az[i] + az[v1]) * (ay[mypz] + ay[v1]));
    advZ += idz * ((az[v5] + az[i]) * (az[v5] + az[i]) - (az[i] + az[v0]) * (az[i] + az[v0]));
    advZ = 0.25 * dt * advZ;
    wx -= advX;
    wy -= advY;
    wz -= advZ;
    auto trace = [&](int c) { return Rn[c] + Rn[c + 3 * n] + Rn[c + 5 * n]; };
    wx += idx * f1 * (Rn[v3] - trace(v3) / 3.);
    wy += idy * f1 * (Rn[v4 + 3 * n] - trace(v4) / 3.);
    wz += idz * f1 * (Rn[v5 + 5 * n] - trace(v5) / 3.);
    wx += idy * f4 * Rn[i + n];
    wy += idx * f4 * Rn[i + n];
    wx += idz * f4 * Rn[i + 2 * n];
    wz += idx * f4 * Rn[i + 2 * n];
    wy += idz * f4 * Rn[i + 4 * n];
    wz += idy * f4 * Rn[i + 4 * n];
    const double tr = trace(i);
    wx -= idx * f1 * (Rn[i] - tr / 3.);
    wy -= idy * f1 * (Rn[i + 3 * n] - tr / 3.);
    wz -= idz * f1 * (Rn[i + 5 * n] - tr / 3.);
    wx -= idy * f4 * Rn[v1 + n];
    wx -= idz * f4 * Rn[v0 + 2 * n];
    wy -= idx * f4 * Rn[v2 + n];
    wy -= idz * f4 * Rn[v0 + 4 * n];
    wz -= idx * f4 * Rn[v2 + 2 * n];
    wz -= idy * f4 * Rn[v1 + 4 * n];
    R.w64[i] = wx;
    R.w64[n + i] = wy;
    R.w64[2 * n + i] = wz;
  }
}

// The transform's real field = u (src/realToComplex.cu:21-38)
template <bool ONE>
__global__ void k_inc_load(FSL_KARGS) {
  FSL_REP_AT(blockIdx.y);
  const size_t n3 = 3 * (size_t)P.nc;
  for (size_t k = blockIdx.x * (size_t)blockDim.x + threadIdx.x; k < n3; k += (size_t)gridDim.x * blockDim.x)
    R.w64[k] = R.v64[k];
}

unsigned cell_blocks(const Batch& B, long work) {
  unsigned bc = blocks_for(work, 256);
  const unsigned cap = (unsigned)((148 * 16 + B.nrep - 1) / B.nrep);
  return bc > cap ? (cap < 1 ? 1 : cap) : bc;
}

}  // namespace

void launch_inc_w(const Batch& B, int second, cudaStream_t s) {
  FSL_GO(k_inc_w, dim3(cell_blocks(B, B.nc), B.nrep), 256, 0, s, B, second);
}

void launch_inc_load(const Batch& B, cudaStream_t s) {
  FSL_GO(k_inc_load, dim3(cell_blocks(B, 3L * B.nc), B.nrep), 256, 0, s, B);
}

}  // namespace fsl
