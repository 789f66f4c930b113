// fsl_fft_cube.cuh -- the whole solve of a small cube in one launch (included
// by fsl_fft.cu after fsl_fft_reg.cuh).
//
// At edges 16 and 24 the four launches of a single instance's solve (W build,
// forward planes, z lines with the solve, inverse planes) are latency: each
// moves a few hundred KB through the L2 in a handful of blocks.  Here a
// cluster of kCubeRanks blocks holds the half spectrum in its shared memory:
// every rank builds W of its 3 N / kCubeRanks planes (and clears the spread
// field behind the read), transforms them, takes its share of the (kx, ky)
// columns from all ranks' planes through distributed shared memory for the z
// transform, the solve and the way back, and finishes its planes.  Two
// cluster barriers, no spectrum or W in global memory.  Back to back, W build
// apart: edge 16 8.4 us against 12.9 for the three passes, edge 24 18.0
// against 20.5; at edge 32 (23.3 against 19.5) the eight SMs no longer keep up.
// A batch keeps the passes although it would gain on its own (64 instances of
// edge 16: 14.3 against 25.8 us): beside the other size classes of a mixed
// batch the clusters wait for eight free blocks at a time (256 mixed
// replicas: 2973 against 2811 us a step).
//
// A line's N points stay in one thread's registers (the N x 1 split of the
// passes).  The line transforms, the packing of columns 0 and N/2, the solve
// and W are the arithmetic of k_plane_fwd_r, k_zsolve_r, k_plane_inv_r and
// k_wbuild4: the same bits, alone and in a batch.

constexpr int kCubeRanks = 8;

template <int N>
struct CubeGeom {
  using G = LineGeom<N, 1>;
  static constexpr int H = N / 2, MXH = H + 1;
  static constexpr int PPR = 3 * N / kCubeRanks;    // planes per rank
  static constexpr int CPR = MXH * N / kCubeRanks;  // (kx, ky) columns per rank
  static constexpr int PB = plane_buf<N, N, 1>();
  static constexpr int NLZ = 3 * CPR;               // z lines per rank
  static constexpr int LINES = PPR * H > NLZ ? PPR * H : NLZ;
  static constexpr int THREADS = LINES < 128 ? 128 : (LINES + 31) / 32 * 32;
  // float2: planes or z lines | half spectrum of the rank's planes
  static constexpr int WORK = PPR * PB > NLZ * G::LS ? PPR * PB : NLZ * G::LS;
  static constexpr int SMEM = WORK + PPR * N * MXH;
  static_assert(3 * N % kCubeRanks == 0 && MXH * N % kCubeRanks == 0 && N % 4 == 0, "equal shares");
  static_assert(2 * PB >= N * (N + 1), "the real plane fits the line buffer");
};

template <int N>
__global__ void __launch_bounds__(CubeGeom<N>::THREADS)
    k_solve_cube(const __grid_constant__ Rep R, const float* __restrict__ sx, const float* __restrict__ sy, const float* __restrict__ sz,
                 const float2* __restrict__ ex, const float2* __restrict__ ey, const float2* __restrict__ ez, const WSrc ws) {
  fsl_pdl_enter();
  if (!R.active) return;  // (all ranks alike)
  const Params& P = R.P;
  namespace cg = cooperative_groups;
  using C = CubeGeom<N>;
  using G = typename C::G;
  constexpr int H = C::H, MXH = C::MXH, PPR = C::PPR, CPR = C::CPR, PB = C::PB, NLZ = C::NLZ, LS = G::LS;
  extern __shared__ __align__(16) float2 smem[];
  float2* work = smem;
  float2* sp = work + C::WORK;  // [plane][ky][kx]
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)blockIdx.x;
  // ---- W of the rank's planes, which are consecutive in memory, into real
  // planes of row pitch N + 1
  {
    const size_t first = (size_t)rank * PPR * N * N;
    constexpr int U = 4;
    for (int g0 = threadIdx.x; g0 < PPR * N * N / 4; g0 += U * blockDim.x)
      w_cells4<U>(
          P, R, ws, [&](int u) { const int i = 4 * (g0 + u * (int)blockDim.x); return i < PPR * N * N ? (long)(first + i) : -1L; },
          [&](int u, float4 w) {
            const int i = 4 * (g0 + u * (int)blockDim.x), lp = i / (N * N), row = i % (N * N) / N, x = i % N;
            float* f = reinterpret_cast<float*>(work + lp * PB) + row * (N + 1) + x;
            f[0] = w.x;
            f[1] = w.y;
            f[2] = w.z;
            f[3] = w.w;
          });
  }
  __syncthreads();
  const int lp = threadIdx.x / H, c = threadIdx.x - lp * H;  // row pair c, then column c, of plane lp
  const bool on = lp < PPR;
  float2* buf = work + (on ? lp : 0) * PB;
  float2 v[N];
  // ---- x forward
  if (on) {
    const float* fw = reinterpret_cast<const float*>(buf);
#pragma unroll
    for (int x = 0; x < N; ++x) v[x] = make_float2(fw[(2 * c) * (N + 1) + x], fw[(2 * c + 1) * (N + 1) + x]);
  }
  __syncthreads();
  if (on) {
    RDft<N>::run(v, -1);
#pragma unroll
    for (int f = 0; f < N; ++f) buf[c * LS + f] = v[f];
  }
  __syncthreads();
  // ---- y forward into the half spectrum
  if (on) {
#pragma unroll
    for (int y = 0; y < N; ++y) {
      const int q = y >> 1, odd = y & 1;
      if (c == 0) {
        const float2 a = buf[q * LS], b = buf[q * LS + H];
        v[y] = odd ? make_float2(a.y, b.y) : make_float2(a.x, b.x);
      } else {
        const float2 zk = buf[q * LS + c], zm = buf[q * LS + N - c];
        v[y] = odd ? make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x))
                   : make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
      }
    }
  }
  __syncthreads();
  float2* pl = sp + (on ? lp : 0) * N * MXH;
  // the packed column: C = F0 + i FH, F0 = (C + conj C-)/2, FH = (C - conj C-)/(2i)
  auto unpack = [&](int f, float2 Cf, float2 Cm) {
    pl[f * MXH] = make_float2(0.5f * (Cf.x + Cm.x), 0.5f * (Cf.y - Cm.y));
    pl[f * MXH + H] = make_float2(0.5f * (Cf.y + Cm.y), -0.5f * (Cf.x - Cm.x));
  };
  if (on) {
    RDft<N>::run(v, -1);
#pragma unroll
    for (int f = 0; f < N; ++f) {
      if (c != 0) pl[f * MXH + c] = v[f];
      else unpack(f, v[f], v[(N - f) % N]);
    }
  }
  cl.sync();
  // ---- z lines of the rank's columns, the solve, and back
  {
    const int l = threadIdx.x % NLZ;
    const bool zon = threadIdx.x < NLZ;
    const int comp = l / CPR, cc = l - comp * CPR, col = rank * CPR + cc;
    float2* lb = work + l * LS;
    // element z of this line: plane comp N + z of its rank
    auto at = [&](int z) {
      const int pz = comp * N + z, rk = pz / PPR;
      return cl.map_shared_rank(sp, rk) + (pz - rk * PPR) * N * MXH + col;
    };
    if (zon) {
#pragma unroll
      for (int k = 0; k < N; ++k) v[k] = *at(k);
      RDft<N>::run(v, -1);
#pragma unroll
      for (int f = 0; f < N; ++f) lb[f] = v[f];
    }
    __syncthreads();
    {
      const float inv_eta = (float)(1.0 / P.eta), inv_nc = 1.0f / (float)P.nc;
      const float tdx = (float)(2.0 * P.invdx), tdy = (float)(2.0 * P.invdy), tdz = (float)(2.0 * P.invdz);
      for (int e = threadIdx.x; e < CPR * N; e += blockDim.x) {
        const int mc = e % CPR, kz = e / CPR, mcol = rank * CPR + mc, mkx = mcol % MXH, mky = mcol / MXH;
        float2* pc[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) pc[a] = work + (a * CPR + mc) * LS + kz;
        const float2 E[3] = {__ldg(ex + mkx), __ldg(ey + mky), __ldg(ez + kz)};
        const float g[3] = {tdx * __ldg(sx + mkx), tdy * __ldg(sy + mky), tdz * __ldg(sz + kz)};
        if (mcol == 0 && kz == 0) {
#pragma unroll
          for (int a = 0; a < 3; ++a) *pc[a] = make_float2(0.f, 0.f);
          continue;
        }
        float2 W[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float2 w = *pc[a];
          W[a] = make_float2(w.x * E[a].x + w.y * E[a].y, w.y * E[a].x - w.x * E[a].y);
        }
        const float G2 = g[0] * g[0] + g[1] * g[1] + g[2] * g[2];
        const float invG2 = 1.0f / G2;
        const float2 GW = make_float2(g[0] * W[0].x + g[1] * W[1].x + g[2] * W[2].x,
                                      g[0] * W[0].y + g[1] * W[1].y + g[2] * W[2].y);
        const float fac = inv_eta * invG2 * inv_nc;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float2 V = make_float2((W[a].x - g[a] * GW.x * invG2) * fac, (W[a].y - g[a] * GW.y * invG2) * fac);
          *pc[a] = make_float2(V.x * E[a].x - V.y * E[a].y, V.y * E[a].x + V.x * E[a].y);
        }
      }
    }
    __syncthreads();
    if (zon) {
#pragma unroll
      for (int k = 0; k < N; ++k) v[k] = lb[k];
    }
    __syncthreads();
    if (zon) {
      RDft<N>::run(v, +1);
#pragma unroll
      for (int k = 0; k < N; ++k) *at(k) = v[k];
    }
  }
  cl.sync();  // (no rank touches another's shared memory after this)
  // ---- y inverse
  constexpr int PR = MXH, PRF = N + 1;
  static_assert(N * PR <= PB && N * PRF <= 2 * PB, "plane rows fit the plane buffer");
  if (on) {
#pragma unroll
    for (int ky = 0; ky < N; ++ky) {
      if (c == 0) {
        const float2 f0 = pl[ky * MXH], fh = pl[ky * MXH + H];
        v[ky] = make_float2(f0.x - fh.y, f0.y + fh.x);  // F0 + i FH
      } else {
        v[ky] = pl[ky * MXH + c];
      }
    }
  }
  // rows y: X_y[c], or X_y[0] + i X_y[H] for the packed column
  auto put = [&](int y, float2 u) {
    if (c == 0) {
      buf[y * PR] = make_float2(u.x, 0.f);
      buf[y * PR + H] = make_float2(u.y, 0.f);
    } else {
      buf[y * PR + c] = u;
    }
  };
  if (on) {
    RDft<N>::run(v, +1);
#pragma unroll
    for (int y = 0; y < N; ++y) put(y, v[y]);
  }
  __syncthreads();
  // ---- x inverse
  if (on) {
#pragma unroll
    for (int x = 0; x < N; ++x) {
      float2 e, o;
      if (x <= H) {
        e = buf[(2 * c) * PR + x];
        o = buf[(2 * c + 1) * PR + x];
      } else {
        e = buf[(2 * c) * PR + N - x];
        o = buf[(2 * c + 1) * PR + N - x];
        e.y = -e.y;
        o.y = -o.y;
      }
      v[x] = make_float2(e.x - o.y, e.y + o.x);  // X_2c + i X_2c+1
    }
  }
  __syncthreads();
  float* fb = reinterpret_cast<float*>(buf);
  if (on) {
    RDft<N>::run(v, +1);
#pragma unroll
    for (int x = 0; x < N; ++x) {
      fb[(2 * c) * PRF + x] = v[x].x;
      fb[(2 * c + 1) * PRF + x] = v[x].y;
    }
  }
  __syncthreads();
  float* vo = R.v + (size_t)rank * PPR * N * N;
  for (int i = threadIdx.x; i < PPR * N * N; i += blockDim.x) {
    const int q = i / (N * N), row = i % (N * N) / N, x = i % N;
    vo[i] = reinterpret_cast<const float*>(work + q * PB)[row * PRF + x];
  }
}
