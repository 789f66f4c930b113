// fsl_fp64.cu -- the FP64 form of the fluid side (FSL_PRECISION_FP64).
//
// The step of the FP32 kernels with every fluid quantity in double: the
// noise (Box-Muller in FP64 on the same Philox words), spreading with FP64
// atomics, W, the FFT-based Stokes solve and the interpolation.  fluam itself
// is FP64 throughout, so this form carries the reference's own arithmetic on
// the GPU; it is the third form of the precision study.  One thread per
// particle and component for the particle side; the transforms are those of
// fsl_fft_g.cu, the cell list and the forces the shared FP64 kernels of
// fsl_particles.cu.
#include "fsl_internal.cuh"

namespace fsl {

namespace {

unsigned blocks_for(long work, int tb) { return (unsigned)((work + tb - 1) / tb); }

// ------------------------------------------------------------------ noise ---
// Normal deviates 4b .. 4b+3 of draw t: the Philox words and uniforms of
// philox_normal4, radius sqrt(-2 ln u) and angle 2 pi u in FP64.
__device__ __forceinline__ void philox_normal4_f64(uint64_t seed, uint64_t t, uint64_t b,
                                                   double2& lo, double2& hi) {
  uint4 c = make_uint4((uint32_t)b, (uint32_t)(b >> 32), (uint32_t)t, (uint32_t)(t >> 32));
  uint4 r = philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  const double s24 = 5.9604644775390625e-08;  // 2^-24
  const double u0 = (double)(2u * (r.x >> 9) + 1u) * s24;
  const double u1 = (double)(2u * (r.y >> 9) + 1u) * s24;
  const double u2 = (double)(2u * (r.z >> 9) + 1u) * s24;
  const double u3 = (double)(2u * (r.w >> 9) + 1u) * s24;
  const double twopi = 6.283185307179586476925286766559;
  const double ra = sqrt(-2.0 * log(u0)), rb = sqrt(-2.0 * log(u2));
  double sa, ca, sb, cb;
  sincos(twopi * u1, &sa, &ca);
  sincos(twopi * u3, &sb, &cb);
  lo = make_double2(ra * ca, ra * sa);
  hi = make_double2(rb * cb, rb * sb);
}

template <bool ONE>
__global__ void k_noise64(FSL_KARGS) {
  FSL_REP_AT(blockIdx.y);
  const uint64_t t = *R.t;
  const uint64_t nb = (P.noise_n + 3) >> 2;
  double2* out = reinterpret_cast<double2*>(R.noise64);
  for (uint64_t b = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; b < nb;
       b += (uint64_t)gridDim.x * blockDim.x) {
    double2 lo, hi;
    philox_normal4_f64(P.seed, t, b, lo, hi);
    out[2 * b] = lo;
    out[2 * b + 1] = hi;
  }
}

// --------------------------------------------------------------- stencils ---
// 3-point kernel of src/deltaGPU.cu:57-68, with its single-precision square
// root of a double argument.
__device__ __forceinline__ double delta3d(double x) {
  x = fabs(x);
  if (x > 1.5) return 0.0;
  if (x < 0.5) return (1. + (double)sqrtf((float)(1. - 3. * x * x))) / 3.;
  return (5. - 3. * x - (double)sqrtf((float)(1. - 3. * (1. - x) * (1. - x)))) / 6.;
}

// 4-point kernel (Peskin, Acta Numerica 2002), the form of delta4f in FP64.
__device__ __forceinline__ double delta4d(double x) {
  x = fabs(x);
  if (x >= 2.0) return 0.0;
  if (x <= 1.0) return (3. - 2. * x + sqrt(1. + 4. * x - 4. * x * x)) / 8.;
  return (5. - 2. * x - sqrt(fmax(-7. + 12. * x - 4. * x * x, 0.0))) / 8.;
}

struct Stencil64 {
  int j0[3];
  double w[3][4];
};

// Stencil of component comp: the node choice of stencil_node (posc) and the
// weights in FP64 (posw).
__device__ __forceinline__ void stencil64(const Params& P, int comp, const double posc[3],
                                          const double posw[3], Stencil64& st) {
  const int m[3] = {P.mx, P.my, P.mz};
  const double h[3] = {P.dx, P.dy, P.dz};
  const double invd[3] = {P.invdx, P.invdy, P.invdz};
  const double L[3] = {P.lx, P.ly, P.lz};
  const double invL[3] = {P.invlx, P.invly, P.invlz};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double off = (d == comp) ? __dmul_rn(0.5, h[d]) : 0.0;
    if (P.kernel == 3) {
      double r = minimage(__dsub_rn(posc[d], off), invL[d], L[d]);
      st.j0[d] = wrap_add(cellidx(r, invd[d], m[d]), -1, m[d]);
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        int j = wrap_add(st.j0[d], k, m[d]);
        double node = ((double)j + 0.5) * h[d] - 0.5 * L[d];
        double rr = minimage((posw[d] - node) - off, invL[d], L[d]);
        st.w[d][k] = delta3d(rr * invd[d]);
      }
      st.w[d][3] = 0.0;
    } else {
      double r = minimage(__dsub_rn(__dsub_rn(posc[d], off), __dmul_rn(0.5, h[d])), invL[d], L[d]);
      st.j0[d] = wrap_add(cellidx(r, invd[d], m[d]), -1, m[d]);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        int j = (st.j0[d] + k) % m[d];
        double node = ((double)j + 0.5) * h[d] - 0.5 * L[d] + off;
        st.w[d][k] = delta4d(minimage(posw[d] - node, invL[d], L[d]) * invd[d]);
      }
    }
  }
}

template <int KN>
__device__ __forceinline__ void spread64_one(const Params& P, int comp, const double posc[3],
                                             const double posw[3], double val,
                                             double* __restrict__ g) {
  Stencil64 st;
  stencil64(P, comp, posc, posw, st);
  double* gc = g + (size_t)comp * P.nc;
#pragma unroll
  for (int c = 0; c < KN; ++c) {
    const int z = (st.j0[2] + c) % P.mz;
#pragma unroll
    for (int b = 0; b < KN; ++b) {
      const int y = (st.j0[1] + b) % P.my;
      const double wyz = st.w[1][b] * st.w[2][c] * val;
      const size_t row = (size_t)P.mx * (y + (size_t)P.my * z);
#pragma unroll
      for (int a = 0; a < KN; ++a) {
        const double v = st.w[0][a] * wyz;
        if (v != 0.0) atomicAdd(gc + row + (st.j0[0] + a) % P.mx, v);
      }
    }
  }
}

// ---------------------------------------------------------------- spread ---
// Eight threads per particle: thread s < 3 spreads component s of the force,
// 3 <= s < 6 (drift modes) component s-3 of the RFD drift (both signs).
// drift: 0 F at q; 1 F at q^{n+1/2} + drift; 2 F at q + drift.  The field is
// the FP64 view of the 8-byte spread buffer; W's build divides by dV.
template <bool ONE, int KN>
__global__ void k_spread64(FSL_KARGS, int drift) {
  FSL_REP_FLAT(KIND_T8);
  const long t = blk * (long)blockDim.x + threadIdx.x;
  const int i = (int)(t >> 3), sub = (int)(t & 7);
  const int np = P.np;
  if (i >= np || sub >= (drift ? 6 : 3)) return;
  double* g = reinterpret_cast<double*>(R.grid);
  if (sub < 3) {
    const double* qf = drift == 1 ? R.qp : R.q;
    const double pos[3] = {qf[i], qf[np + i], qf[2 * (size_t)np + i]};
    spread64_one<KN>(P, sub, pos, pos, R.F[(size_t)sub * np + i], g);
    return;
  }
  const int comp = sub - 3;
  const size_t wb = (size_t)6 * P.nc;
  const double W[3] = {R.noise64[wb + i], R.noise64[wb + np + i], R.noise64[wb + 2 * (size_t)np + i]};
  const double pos[3] = {R.q[i], R.q[np + i], R.q[2 * (size_t)np + i]};
  double pp[3], pm[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    pp[d] = pos[d] + 0.5 * kRfdDelta * W[d];
    pm[d] = pos[d] - 0.5 * kRfdDelta * W[d];
  }
  const double vp = (P.kT / kRfdDelta) * W[comp], vm = (P.kT / kRfdDelta) * -1 * W[comp];
  // reference mode: nodes from the displaced position, weights at q
  spread64_one<KN>(P, comp, pp, P.rfd == 1 ? pp : pos, vp, g);
  spread64_one<KN>(P, comp, pm, P.rfd == 1 ? pm : pos, vm, g);
}

// ------------------------------------------------------------------- W ---
// W = f / dV + nfac div(Sigma) per cell (the formulas of k_wbuild in FP64),
// into the transform's real field; the spread field is cleared behind the
// read.
template <bool ONE>
__global__ void k_wbuild64(FSL_KARGS, int nsets, double nfac) {
  FSL_REP_AT(blockIdx.y);
  const size_t nc = (size_t)P.nc;
  const int mx = P.mx, my = P.my, mz = P.mz;
  const double inv_dV = 1.0 / P.dV;
  const double f1 = nfac * P.fact1, f4 = nfac * P.fact4;
  const double a1x = P.invdx * f1, a1y = P.invdy * f1, a1z = P.invdz * f1;
  const double a4x = P.invdx * f4, a4y = P.invdy * f4, a4z = P.invdz * f4;
  double* g = reinterpret_cast<double*>(R.grid);
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nc;
       i += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % mx), r = (int)(i / mx);
    const int y = r % my, z = r / my;
    const int xm = x == 0 ? mx - 1 : x - 1, xp = x == mx - 1 ? 0 : x + 1;
    const int ym = y == 0 ? my - 1 : y - 1, yp = y == my - 1 ? 0 : y + 1;
    const int zm = z == 0 ? mz - 1 : z - 1, zp = z == mz - 1 ? 0 : z + 1;
    const size_t rowyz = (size_t)mx * (y + (size_t)my * z);
    const size_t v0 = x + (size_t)mx * (y + (size_t)my * zm), v1 = x + (size_t)mx * (ym + (size_t)my * z),
                 v2 = xm + rowyz, v3 = xp + rowyz, v4 = x + (size_t)mx * (yp + (size_t)my * z),
                 v5 = x + (size_t)mx * (y + (size_t)my * zp);
    double w[3] = {g[i] * inv_dV, g[nc + i] * inv_dV, g[2 * nc + i] * inv_dV};
    for (int set = 0; set < nsets; ++set) {
      const double* d = R.noise64 + (set ? (size_t)6 * nc + (size_t)9 * P.np : 0);
      w[0] += a1x * (d[v3] - d[i]) + a4y * (d[nc + i] - d[nc + v1]) + a4z * (d[2 * nc + i] - d[2 * nc + v0]);
      w[1] += a1y * (d[3 * nc + v4] - d[3 * nc + i]) + a4x * (d[nc + i] - d[nc + v2]) +
              a4z * (d[4 * nc + i] - d[4 * nc + v0]);
      w[2] += a1z * (d[5 * nc + v5] - d[5 * nc + i]) + a4x * (d[2 * nc + i] - d[2 * nc + v2]) +
              a4y * (d[4 * nc + i] - d[4 * nc + v1]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      R.w64[c * nc + i] = w[c];
      g[c * nc + i] = 0.0;
    }
  }
}

// ------------------------------------------------------ interpolation ---
// Eight threads per particle, thread s < 3 interpolates component s and
// updates that coordinate: stage 1 q^{n+1/2} = q^n + dt/2 J(q^n) v, stage 2
// q^{n+1} = q^n + dt J(q^{n+1/2}) v, each with the extraMobility terms
// (src/stokesLimitFunctions.cu:2646-2650, 3676-3681).
template <bool ONE, int KN>
__global__ void k_interp_update64(FSL_KARGS, int stage) {
  FSL_REP_FLAT(KIND_T8);
  const long t = blk * (long)blockDim.x + threadIdx.x;
  const int i = (int)(t >> 3), comp = (int)(t & 7);
  const int np = P.np;
  if (i >= np || comp >= 3) return;
  const double* qpos = stage == 1 ? R.q : R.qp;
  double* qout = stage == 1 ? R.qp : R.q;
  const double pos[3] = {qpos[i], qpos[np + i], qpos[2 * (size_t)np + i]};
  Stencil64 st;
  stencil64(P, comp, pos, pos, st);
  const double* vc = R.v64 + (size_t)comp * P.nc;
  double u = 0.0;
#pragma unroll
  for (int a = 0; a < KN; ++a) {
    const int x = (st.j0[0] + a) % P.mx;
#pragma unroll
    for (int b = 0; b < KN; ++b) {
      const int y = (st.j0[1] + b) % P.my;
#pragma unroll
      for (int c = 0; c < KN; ++c) {
        const int z = (st.j0[2] + c) % P.mz;
        u += st.w[0][a] * st.w[1][b] * st.w[2][c] * vc[x + (size_t)P.mx * (y + (size_t)P.my * z)];
      }
    }
  }
  const size_t k = (size_t)comp * np + i;
  const double h = stage == 1 ? 0.5 * P.dt : P.dt;
  double r = R.q[k] + h * u;
  if (P.has_extra) {
    const size_t nb = (size_t)6 * P.nc + (size_t)(3 + comp) * np + i;
    double xi = R.noise64[nb];
    if (stage == 2) xi += R.noise64[nb + (size_t)3 * np];
    r += h * P.extra_mob * R.F[k] + P.fact2 * xi;
  }
  if (!isfinite(r)) set_err(R.err, 2);
  qout[k] = r;
}

}  // namespace

// ---------------------------------------------------------------- launchers
void launch_noise64(const Batch& B, cudaStream_t s) {
  const int tb = 256;
  const uint64_t nb = (B.max_noise_n + 3) / 4;
  unsigned bx = blocks_for((long)nb, tb);
  const unsigned cap = (unsigned)((148 * 16 + B.nrep - 1) / B.nrep);
  if (bx > cap) bx = cap < 1 ? 1 : cap;
  FSL_GO(k_noise64, dim3(bx, B.nrep), tb, 0, s, B);
}

void launch_spread64(const Batch& B, int drift, cudaStream_t s) {
  if (B.max_np == 0) return;
  const unsigned g = part_blocks(B, KIND_T8);
  if (B.kernel == 4)
    FSL_GO_T(k_spread64, 4, g, kPartThreads, 0, s, B, drift);
  else
    FSL_GO_T(k_spread64, 3, g, kPartThreads, 0, s, B, drift);
}

void launch_interp_update64(const Batch& B, int stage, cudaStream_t s) {
  if (B.max_np == 0) return;
  const unsigned g = part_blocks(B, KIND_T8);
  if (B.kernel == 4)
    FSL_GO_T(k_interp_update64, 4, g, kPartThreads, 0, s, B, stage);
  else
    FSL_GO_T(k_interp_update64, 3, g, kPartThreads, 0, s, B, stage);
}

void launch_solve64(const Batch& B, const GPlan* g, int nsets, double nfac, cudaStream_t s, Prof* prof) {
  const int tb = 256;
  unsigned bc = blocks_for((long)B.nc, tb);
  const unsigned cap = (unsigned)((148 * 16 + B.nrep - 1) / B.nrep);
  if (bc > cap) bc = cap < 1 ? 1 : cap;
  if (prof) prof->mark(s, "wbuild64");
  FSL_GO(k_wbuild64, dim3(bc, B.nrep), tb, 0, s, B, nsets, nfac);
  if (prof) prof->mark(s, "fft64");
  int n = launch_g_forward(B, g, 3, s);
  if (prof) prof->mark(s, "solve64");
  launch_g_z(B, g, 0, s);
  if (prof) prof->mark(s, "fft64");
  n += launch_g_inverse(B, g, 3, 0, 1.0, s);
  if (prof) prof->count(2 + n);
}

}  // namespace fsl
