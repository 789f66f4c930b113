// fsl_fp64.cu -- the FP64 form of the fluid side (FSL_PRECISION_FP64).
//
// The step of the FP32 kernels with every fluid quantity in double: the
// noise (Box-Muller in FP64 on the same Philox words), spreading with FP64
// atomics, W, the FFT-based Stokes solve and the interpolation.  fluam itself
// is FP64 throughout, so this form carries the reference's own arithmetic on
// the GPU; it is the third form of the precision study.  One warp per
// particle for the spread and the interpolation; the transforms are those of
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

// The spread and the interpolation take one warp per particle: lane
// (f 3 + d) KN + k computes node k of family f (0: cell centres, 1: faces) in
// dimension d, the nodes go round by shuffles, and lane a + 4 b + 16 c0
// handles the x node a, the y node b and the z nodes c0, c0 + 2 of every
// component.  (A thread per particle and component, each with the whole
// stencil of its component in sequence, took 51 us for a spread of 4,096
// particles and 20 us for an interpolation: one serial chain of FP64 weights
// and 64 products.)
struct Lane64 {
  int j;
  double w;
};

// The node choice of stencil_node (posc) and the weight in FP64 (posw).
template <int KN>
__device__ __forceinline__ Lane64 lane64(const Params& P, const double posc[3], const double posw[3], int lane) {
  Lane64 s{0, 0.0};
  if (lane >= 6 * KN) return s;
  const int k = lane % KN, fd = lane / KN, f = fd / 3, d = fd - 3 * f;
  const double pc = d == 0 ? posc[0] : (d == 1 ? posc[1] : posc[2]);
  const double pw = d == 0 ? posw[0] : (d == 1 ? posw[1] : posw[2]);
  const int m = d == 0 ? P.mx : (d == 1 ? P.my : P.mz);
  const double h = d == 0 ? P.dx : (d == 1 ? P.dy : P.dz);
  const double invd = d == 0 ? P.invdx : (d == 1 ? P.invdy : P.invdz);
  const double L = d == 0 ? P.lx : (d == 1 ? P.ly : P.lz);
  const double invL = d == 0 ? P.invlx : (d == 1 ? P.invly : P.invlz);
  const double off = f ? __dmul_rn(0.5, h) : 0.0;
  double r = __dsub_rn(pc, off);
  if (KN == 4) r = __dsub_rn(r, __dmul_rn(0.5, h));
  s.j = wrap_add(cellidx(minimage(r, invL, L), invd, m), k - 1, m);
  const double node = ((double)s.j + 0.5) * h - 0.5 * L;
  const double x = minimage((pw - node) - off, invL, L) * invd;
  s.w = KN == 4 ? delta4d(x) : delta3d(x);
  return s;
}

struct Nodes64 {
  int jx[2], jy[2], jz[2][2];
  double wx[2], wy[2], wz[2][2];
  bool on[2];
};

template <int KN>
__device__ __forceinline__ void share64(const Lane64& s, int lane, Nodes64& N) {
  const unsigned full = 0xffffffffu;
  const int a = lane & 3, b = (lane >> 2) & 3, c0 = lane >> 4;
  const int ka = min(a, KN - 1), kb = min(b, KN - 1), kc = min(c0 + 2, KN - 1);
#pragma unroll
  for (int f = 0; f < 2; ++f) {
    const int at = 3 * f * KN;
    N.jx[f] = __shfl_sync(full, s.j, at + ka);
    N.wx[f] = __shfl_sync(full, s.w, at + ka);
    N.jy[f] = __shfl_sync(full, s.j, at + KN + kb);
    N.wy[f] = __shfl_sync(full, s.w, at + KN + kb);
    N.jz[f][0] = __shfl_sync(full, s.j, at + 2 * KN + c0);
    N.wz[f][0] = __shfl_sync(full, s.w, at + 2 * KN + c0);
    N.jz[f][1] = __shfl_sync(full, s.j, at + 2 * KN + kc);
    N.wz[f][1] = __shfl_sync(full, s.w, at + 2 * KN + kc);
  }
  N.on[0] = a < KN && b < KN;
  N.on[1] = N.on[0] && c0 + 2 < KN;
}

__device__ __forceinline__ void spread64_one(const Params& P, const Nodes64& N, const double val[3], double* __restrict__ g) {
#pragma unroll
  for (int comp = 0; comp < 3; ++comp) {
    if (val[comp] == 0.0) continue;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (!N.on[c]) continue;
      const double v = N.wx[comp == 0] * (N.wy[comp == 1] * N.wz[comp == 2][c] * val[comp]);
      if (v != 0.0)
        atomicAdd(g + (size_t)comp * P.nc + (N.jx[comp == 0] + (size_t)P.mx * (N.jy[comp == 1] + (size_t)P.my * N.jz[comp == 2][c])), v);
    }
  }
}

// ---------------------------------------------------------------- spread ---
// drift: 0 F at q; 1 F at q^{n+1/2} + the RFD drift at q; 2 F and the drift
// at q.  The field is the FP64 view of the 8-byte spread buffer; W's build
// divides by dV.  In reference mode the drift's nodes come from the displaced
// positions and its weights from q: the spreads of the two signs cancel for
// every component whose nodes are the same, which is left out.
template <bool ONE, int KN>
__global__ void __launch_bounds__(kPartThreads) k_spread64(FSL_KARGS, int drift) {
  FSL_REP_FLAT(KIND_T32);
  const long e = (blk * (long)blockDim.x + threadIdx.x) >> 5;
  const int np = P.np, lane = threadIdx.x & 31;
  if (e >= np) return;  // a whole warp
  const int i = (int)e;
  double* g = reinterpret_cast<double*>(R.grid);
  Nodes64 N;
  {
    const double* qf = drift == 1 ? R.qp : R.q;
    const double pos[3] = {qf[i], qf[np + i], qf[2 * (size_t)np + i]};
    const double val[3] = {R.F[i], R.F[np + i], R.F[2 * (size_t)np + i]};
    share64<KN>(lane64<KN>(P, pos, pos, lane), lane, N);
    spread64_one(P, N, val, g);
  }
  if (!drift) return;
  const size_t wb = (size_t)6 * P.nc;
  const double W[3] = {R.noise64[wb + i], R.noise64[wb + np + i], R.noise64[wb + 2 * (size_t)np + i]};
  const double pos[3] = {R.q[i], R.q[np + i], R.q[2 * (size_t)np + i]};
  double pp[3], pm[3], vp[3], vm[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    pp[d] = pos[d] + 0.5 * kRfdDelta * W[d];
    pm[d] = pos[d] - 0.5 * kRfdDelta * W[d];
    vp[d] = (P.kT / kRfdDelta) * W[d];
    vm[d] = (P.kT / kRfdDelta) * -1 * W[d];
  }
  if (P.rfd != 1) {
    bool diff = false;
    if (lane < 6) {
      const int f = lane / 3, d = lane - 3 * f;
      diff = stencil_base(P, d, f, d == 0 ? pp[0] : (d == 1 ? pp[1] : pp[2])) !=
             stencil_base(P, d, f, d == 0 ? pm[0] : (d == 1 ? pm[1] : pm[2]));
    }
    const unsigned chg = __ballot_sync(0xffffffffu, diff);
    if (!chg) return;  // the whole warp
    constexpr unsigned fam[3] = {(1 << 3) | (1 << 1) | (1 << 2), (1 << 4) | (1 << 0) | (1 << 2), (1 << 5) | (1 << 0) | (1 << 1)};
#pragma unroll
    for (int c = 0; c < 3; ++c)
      if (!(chg & fam[c])) vp[c] = vm[c] = 0.0;
  }
  share64<KN>(lane64<KN>(P, pp, P.rfd == 1 ? pp : pos, lane), lane, N);
  spread64_one(P, N, vp, g);
  share64<KN>(lane64<KN>(P, pm, P.rfd == 1 ? pm : pos, lane), lane, N);
  spread64_one(P, N, vm, g);
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
// Stage 1 q^{n+1/2} = q^n + dt/2 J(q^n) v, stage 2 q^{n+1} = q^n + dt
// J(q^{n+1/2}) v, each with the extraMobility terms
// (src/stokesLimitFunctions.cu:2646-2650, 3676-3681).
template <bool ONE, int KN>
__global__ void __launch_bounds__(kPartThreads) k_interp_update64(FSL_KARGS, int stage) {
  FSL_REP_FLAT(KIND_T32);
  const long e = (blk * (long)blockDim.x + threadIdx.x) >> 5;
  const int np = P.np, lane = threadIdx.x & 31;
  if (e >= np) return;  // a whole warp
  const int i = (int)e;
  const double* qpos = stage == 1 ? R.q : R.qp;
  double* qout = stage == 1 ? R.qp : R.q;
  const double pos[3] = {qpos[i], qpos[np + i], qpos[2 * (size_t)np + i]};
  Nodes64 N;
  share64<KN>(lane64<KN>(P, pos, pos, lane), lane, N);
  double us[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double u = 0.0;
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (N.on[c])
        u += N.wx[d == 0] * N.wy[d == 1] * N.wz[d == 2][c] *
             R.v64[(size_t)d * P.nc + (N.jx[d == 0] + (size_t)P.mx * (N.jy[d == 1] + (size_t)P.my * N.jz[d == 2][c]))];
    us[d] = u;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int d = 0; d < 3; ++d) us[d] += __shfl_xor_sync(0xffffffffu, us[d], o);
  const int comp = lane < 3 ? lane : 0;  // the other lanes join the shuffles
  const size_t k = (size_t)comp * np + i;
  const double h = stage == 1 ? 0.5 * P.dt : P.dt;
  double r = R.q[k] + h * (comp == 0 ? us[0] : (comp == 1 ? us[1] : us[2]));
  if (P.has_extra) {
    const size_t nb = (size_t)6 * P.nc + (size_t)(3 + comp) * np + i;
    double xi = R.noise64[nb];
    if (stage == 2) xi += R.noise64[nb + (size_t)3 * np];
    r += h * P.extra_mob * R.F[k] + P.fact2 * xi;
  }
  if (P.verlet) {
    // a particle beyond half the skin from its reference position: the list
    // is rebuilt at the next evaluation (k_interp_update)
    const double d = lane < 3 ? r - R.qref[k] : 0.0;
    double d2 = d * d;
    d2 += __shfl_xor_sync(0xffffffffu, d2, 1);
    d2 += __shfl_xor_sync(0xffffffffu, d2, 2);
    if (lane == 0 && d2 > P.vl_half2) R.vl_flag[stage == 1 ? 1 : 0] = *R.t + stage;
  }
  if (lane >= 3) return;
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
  const unsigned g = part_blocks(B, KIND_T32);
  if (B.kernel == 4)
    FSL_GO_T(k_spread64, 4, g, kPartThreads, 0, s, B, drift);
  else
    FSL_GO_T(k_spread64, 3, g, kPartThreads, 0, s, B, drift);
}

void launch_interp_update64(const Batch& B, int stage, cudaStream_t s) {
  if (B.max_np == 0) return;
  const unsigned g = part_blocks(B, KIND_T32);
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
