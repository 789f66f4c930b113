// fsl_fft_g.cu -- the periodic transforms of any 2,3,5,7,11-smooth extents,
// FP32 and FP64: the Stokes solve of grids without compiled passes
// (fsl_fft_reg.cuh), and every transform of the FP64 forms (the FP64 Stokes
// step, the quasi-2D family, the incompressible fluid).
//
// A line of N points is transformed by Stockham stages of large radix
// (at most 16) held in registers: N = r1 r2 with both at most 16 for nearly
// every extent up to 256, three or four stages otherwise.  The radices are
// compiled, everything else is a runtime number: a stage is one switch over
// the radix, so one kernel serves every extent and a line costs one exchange
// through shared memory per extra stage (against four or five with radices
// 4, 2, 3, 5) and one barrier each.  Real fields are transformed as pairs of
// rows (two real rows are one complex line) into the half spectrum
// [comp][z][ky][kx], kx <= mx/2.  Passes:
//   k_g_plane_fwd / k_g_plane_inv  whole xy planes in shared memory, where
//                                  both extents have two stages and it fits;
//   k_g_x_fwd, k_g_y, k_g_x_inv    one axis each, otherwise;
//   k_g_z                          z lines of all components of a (kx, ky)
//                                  tile, the solve of every mode, and back.
// What bounds them: below about 128^3 the data stays in the L2 and a pass is
// a latency chain of its barriers; beyond, the passes stream the spectrum
// through HBM.
#include <cmath>
#include <cstdlib>
#include <vector>

#include <algorithm>
#include "fsl_internal.cuh"

namespace fsl {

namespace {

constexpr int kGRad = 16;    // largest radix
constexpr int kGStages = 4;  // 625 = 5^4 and 875 need four

// One axis: extent n, stage radices f[0..ns).  t = n / f[0] threads hold a
// line (f[0] points each); two stages: f[0] >= f[1] = t.
struct GAxis {
  int n, ns, t;
  int f[kGStages];
};

template <class V>
struct GReal;
template <>
struct GReal<float2> {
  using T = float;
};
template <>
struct GReal<double2> {
  using T = double;
};
template <class V>
using greal = typename GReal<V>::T;

template <class V>
__device__ __forceinline__ V gmk(greal<V> x, greal<V> y) {
  V v;
  v.x = x;
  v.y = y;
  return v;
}
template <class V>
__device__ __forceinline__ V gmul(V a, V b) {
  return gmk<V>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <class V>
__device__ __forceinline__ V gadd(V a, V b) {
  return gmk<V>(a.x + b.x, a.y + b.y);
}
template <class V>
__device__ __forceinline__ V gsub(V a, V b) {
  return gmk<V>(a.x - b.x, a.y - b.y);
}

// exp(-2 pi i j / R), j < R <= 16: read at compile-time indexes
__constant__ float2 c_g32[kGRad + 1][kGRad];
__constant__ double2 c_g64[kGRad + 1][kGRad];

template <class V, int R, int DIR>
__device__ __forceinline__ V groot(int j) {
  V w;
  if constexpr (sizeof(V) == sizeof(float2)) {
    const float2 c = c_g32[R][j % R];
    w = gmk<V>(c.x, c.y);
  } else {
    const double2 c = c_g64[R][j % R];
    w = gmk<V>(c.x, c.y);
  }
  if (DIR > 0) w.y = -w.y;
  return w;
}

// DFT of R points in registers, natural order in and out:
// V[f] = sum_x v[x] exp(DIR 2 pi i f x / R).
template <class V, int R, int DIR>
struct GDft {
  __device__ __forceinline__ static void run(V (&v)[R]) {
    if constexpr (R == 1) {
    } else if constexpr (R == 2) {
      const V a = v[0], b = v[1];
      v[0] = gadd(a, b);
      v[1] = gsub(a, b);
    } else if constexpr (R == 4) {
      const V a = gadd(v[0], v[2]), b = gsub(v[0], v[2]), c = gadd(v[1], v[3]), e = gsub(v[1], v[3]);
      const V d = DIR > 0 ? gmk<V>(-e.y, e.x) : gmk<V>(e.y, -e.x);
      v[0] = gadd(a, c);
      v[2] = gsub(a, c);
      v[1] = gadd(b, d);
      v[3] = gsub(b, d);
    } else if constexpr (R == 3 || R == 5 || R == 7 || R == 11) {
      // sums and differences of the pairs (r, R - r): real factors only
      constexpr int H = R / 2;
      V s[H], d[H];
#pragma unroll
      for (int r = 1; r <= H; ++r) {
        s[r - 1] = gadd(v[r], v[R - r]);
        d[r - 1] = gsub(v[r], v[R - r]);
      }
      const V z = v[0];
#pragma unroll
      for (int r = 0; r < H; ++r) v[0] = gadd(v[0], s[r]);
#pragma unroll
      for (int q = 1; q <= H; ++q) {
        V a = z, b = gmk<V>(0, 0);
#pragma unroll
        for (int r = 1; r <= H; ++r) {
          const V w = groot<V, R, DIR>(r * q);
          a.x += w.x * s[r - 1].x;
          a.y += w.x * s[r - 1].y;
          b.x += w.y * d[r - 1].x;
          b.y += w.y * d[r - 1].y;
        }
        v[q] = gmk<V>(a.x - b.y, a.y + b.x);  // a + i b
        v[R - q] = gmk<V>(a.x + b.y, a.y - b.x);
      }
    } else {
      constexpr int P = R % 4 == 0 ? 4 : R % 2 == 0 ? 2 : R % 3 == 0 ? 3 : R % 5 == 0 ? 5 : 7;
      constexpr int Q = R / P;
      V Y[P][Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        V u[P];
#pragma unroll
        for (int p = 0; p < P; ++p) u[p] = v[q + Q * p];
        GDft<V, P, DIR>::run(u);
#pragma unroll
        for (int g = 0; g < P; ++g) Y[g][q] = g * q == 0 ? u[g] : gmul(u[g], groot<V, R, DIR>(g * q));
      }
#pragma unroll
      for (int g = 0; g < P; ++g) {
        GDft<V, Q, DIR>::run(Y[g]);
#pragma unroll
        for (int h = 0; h < Q; ++h) v[g + P * h] = Y[g][h];
      }
    }
  }
};

template <class V, int DIR, int R, class Ld, class St>
__device__ __forceinline__ void gbfly(Ld&& ld, St&& st) {
  V v[R];
#pragma unroll
  for (int q = 0; q < R; ++q) v[q] = ld(q);
  GDft<V, R, DIR>::run(v);
#pragma unroll
  for (int q = 0; q < R; ++q) st(q, v[q]);
}

// One butterfly of runtime radix r <= RMAX: inputs ld(0 .. r-1), outputs
// st(0 .. r-1, value).
template <class V, int DIR, int RMAX, class Ld, class St>
__device__ __forceinline__ void gstage(int r, Ld&& ld, St&& st) {
  if constexpr (RMAX > 8) {
    switch (r) {
      case 9: gbfly<V, DIR, 9>(ld, st); return;
      case 10: gbfly<V, DIR, 10>(ld, st); return;
      case 11: gbfly<V, DIR, 11>(ld, st); return;
      case 12: gbfly<V, DIR, 12>(ld, st); return;
      case 14: gbfly<V, DIR, 14>(ld, st); return;
      case 15: gbfly<V, DIR, 15>(ld, st); return;
      case 16: gbfly<V, DIR, 16>(ld, st); return;
      default: break;
    }
  }
  switch (r) {
    case 2: gbfly<V, DIR, 2>(ld, st); return;
    case 3: gbfly<V, DIR, 3>(ld, st); return;
    case 4: gbfly<V, DIR, 4>(ld, st); return;
    case 5: gbfly<V, DIR, 5>(ld, st); return;
    case 6: gbfly<V, DIR, 6>(ld, st); return;
    case 7: gbfly<V, DIR, 7>(ld, st); return;
    case 8: gbfly<V, DIR, 8>(ld, st); return;
    default: gbfly<V, DIR, 1>(ld, st); return;
  }
}

template <class V, int DIR>
__device__ __forceinline__ V gtw(const V* __restrict__ tw, int i) {
  V w = tw[i];
  if (DIR > 0) w.y = -w.y;
  return w;
}

// The first and second stage of a two-stage line: thread t < A.t takes the
// points t + A.t k; pos(a, t) is where output a of thread t waits; after a
// barrier, thread t takes the rows a = t, t + A.t, ...
template <class V, int DIR, int RMAX, class Ld, class Pos>
__device__ __forceinline__ void gfirst(const GAxis& A, int t, V* ex, Ld&& ld, Pos&& pos) {
  gstage<V, DIR, RMAX>(
      A.f[0], [&](int k) { return ld(t + A.t * k); }, [&](int a, V v) { ex[pos(a, t)] = v; });
}
template <class V, int DIR, int RMAX, class Pos, class Em>
__device__ __forceinline__ void gsecond(const GAxis& A, int t, const V* ex, const V* __restrict__ tw, Pos&& pos, Em&& emit) {
  for (int a = t; a < A.f[0]; a += A.t)
    gstage<V, DIR, RMAX>(
        A.f[1],
        [&](int tt) {
          const V v = ex[pos(a, tt)];
          return tt == 0 ? v : gmul(v, gtw<V, DIR>(tw, a * tt));
        },
        [&](int b, V v) { emit(a + A.f[0] * b, v); });
}

// A whole line by A.t threads (two stages that emit elsewhere than to the
// other buffer need only b0).  Output a of the first stage's thread t waits
// at pos(a, t) (two stages), point i between more stages at at(i).  Two
// buffers; emit(f, value, other) gets the one that the last stage does not
// read.  All threads of the block call this; `on` ones work.  The caller
// puts a barrier after it before the buffers are written again.
template <class V, int DIR, int RMAX, bool MULTI, class Pos, class At, class Ld, class Em>
__device__ __forceinline__ void gline(const GAxis& A, int t, bool on, V* b0, V* b1, const V* __restrict__ tw, Pos&& pos,
                                      At&& at, Ld&& ld, Em&& emit) {
  if constexpr (!MULTI) {
    if (on) gfirst<V, DIR, RMAX>(A, t, b0, ld, pos);
    __syncthreads();
    if (on) gsecond<V, DIR, RMAX>(A, t, b0, tw, pos, [&](int f, V v) { emit(f, v, b1); });
  } else {
    if (on)
      gstage<V, DIR, RMAX>(
          A.f[0], [&](int k) { return ld(t + A.t * k); }, [&](int a, V v) { b0[at(t * A.f[0] + a)] = v; });
    int Ns = A.f[0];
    V *in = b0, *out = b1;
    for (int s = 1; s < A.ns; ++s) {
      __syncthreads();
      const int r = A.f[s], nb = A.n / r, str = A.n / (Ns * r);
      const bool last = s == A.ns - 1;
      if (on)
        for (int j = t; j < nb; j += A.t) {
          const int k = j % Ns, d = (j - k) * r + k;
          gstage<V, DIR, RMAX>(
              r,
              [&](int q) {
                const V v = in[at(j + q * nb)];
                return q == 0 ? v : gmul(v, gtw<V, DIR>(tw, q * k * str));
              },
              [&](int q, V v) {
                if (last) emit(d + q * Ns, v, out);
                else out[at(d + q * Ns)] = v;
              });
        }
      Ns *= r;
      V* sw = in;
      in = out;
      out = sw;
    }
  }
}

// What the kernels need of an instance: by value for a single one, else read
// from the class's device table.
struct GInst {
  const void* w;   // real field in [comp][z][y][x]
  void* spec;      // half spectrum
  void* v;         // real field out
  const void* u;   // k_g_*_inv with pred: out = (field + u) / 2
  double invdx, invdy, invdz, eta, dt, rho;
  int active;
};

struct GArgs {
  GInst one;
  const Rep* reps;  // null: `one`
  int mx, my, mz, mxh, ncomp;
  int f64, pred;
};

__host__ __device__ inline GInst g_inst_of(const Rep& r, int f64, int pred) {
  GInst g;
  g.active = r.active;
  g.w = f64 ? (const void*)r.w64 : (const void*)r.wbuf;
  g.spec = f64 ? (void*)r.z64 : (void*)r.spec;
  g.v = pred ? (void*)r.grid : f64 ? (void*)r.v64 : (void*)r.v;
  g.u = r.v64;
  g.invdx = r.P.invdx;
  g.invdy = r.P.invdy;
  g.invdz = r.P.invdz;
  g.eta = r.P.eta;
  g.dt = r.P.dt;
  g.rho = r.P.rho;
  return g;
}

__device__ __forceinline__ GInst g_inst(const GArgs& g, int idx) {
  return g.reps ? g_inst_of(g.reps[idx], g.f64, g.pred) : g.one;
}

// Launch numbers of the plane kernels: lines per group (lx row pairs, ly
// columns), shared pitches (elements).
struct GPlane {
  GAxis ax, ay;
  int lx, ly, npairs;
  int nt;         // exchange pitch of the x stage, 1 mod 16 (8 in FP64)
  int pitch;      // plane row (pair) pitch of the forward / inverse kernel
  int ex_off;     // first element of the exchange
  const void *twx, *twy;
  double scale;   // of the inverse's real output
};

// ------------------------------------------------------------ whole planes ---
// One xy plane per block: row pairs as complex lines into Z_p (pitch: T mod
// 16 elements, so that a warp's stores fall on distinct banks), then the
// columns kx <= mx/2, whose points are split from Z_p on the way in
// (X_k = (Z_k + conj Z_-k)/2, Y_k = -i (Z_k - conj Z_-k)/2).
template <class V, int RMAX, int NT>
__global__ void __launch_bounds__(NT) k_g_plane_fwd(const __grid_constant__ GArgs g, const __grid_constant__ GPlane p) {
  fsl_pdl_enter();
  const GInst I = g_inst(g, blockIdx.y);
  if (!I.active) return;
  using T = greal<V>;
  extern __shared__ __align__(16) unsigned char g_smem[];
  V* twx = reinterpret_cast<V*>(g_smem);
  V* twy = twx + g.mx;
  V* pl = twy + g.my;
  V* ex = twx + p.ex_off;
  for (int i = threadIdx.x; i < g.mx; i += blockDim.x) twx[i] = reinterpret_cast<const V*>(p.twx)[i];
  for (int i = threadIdx.x; i < g.my; i += blockDim.x) twy[i] = reinterpret_cast<const V*>(p.twy)[i];
  const int mx = g.mx, my = g.my;
  const T* W = reinterpret_cast<const T*>(I.w) + (size_t)blockIdx.x * mx * my;
  __syncthreads();
  {
    const int l = threadIdx.x / p.ax.t, t = threadIdx.x - l * p.ax.t;
    auto pos = [&](int a, int tt) { return a * p.nt + l * p.ax.t + tt; };
    for (int g0 = 0; g0 < p.npairs; g0 += p.lx) {
      const int pr = g0 + l;
      const bool on = l < p.lx && pr < p.npairs;
      if (on) {
        const T* r0 = W + (size_t)(2 * pr) * mx;
        const bool two = 2 * pr + 1 < my;
        gfirst<V, -1, RMAX>(p.ax, t, ex, [&](int x) { return gmk<V>(r0[x], two ? r0[mx + x] : (T)0); }, pos);
      }
      __syncthreads();
      if (on) gsecond<V, -1, RMAX>(p.ax, t, ex, twx, pos, [&](int f, V v) { pl[pr * p.pitch + f] = v; });
      __syncthreads();
    }
  }
  {
    const int t = threadIdx.x / p.ly, cl = threadIdx.x - t * p.ly;
    V* out = reinterpret_cast<V*>(I.spec) + (size_t)blockIdx.x * my * g.mxh;
    auto pos = [&](int a, int tt) { return (a * p.ay.t + tt) * p.ly + cl; };
    for (int c0 = 0; c0 < g.mxh; c0 += p.ly) {
      const int c = c0 + cl;
      const bool on = t < p.ay.t && c < g.mxh;
      const int cm = c ? mx - c : 0;
      if (on)
        gfirst<V, -1, RMAX>(
            p.ay, t, ex,
            [&](int y) {
              const V* z = pl + (y >> 1) * p.pitch;
              const V zk = z[c], zm = z[cm];
              const T h = (T)0.5;
              return (y & 1) ? gmk<V>(h * (zk.y + zm.y), -h * (zk.x - zm.x)) : gmk<V>(h * (zk.x + zm.x), h * (zk.y - zm.y));
            },
            pos);
      __syncthreads();
      if (on) gsecond<V, -1, RMAX>(p.ay, t, ex, twy, pos, [&](int f, V v) { out[(size_t)f * g.mxh + c] = v; });
      __syncthreads();
    }
  }
}

// The inverse: columns into the half-spectrum plane, then the row pairs with
// the Hermitian completion X[N - x] = conj X[x].
template <class V, int RMAX, int NT>
__global__ void __launch_bounds__(NT) k_g_plane_inv(const __grid_constant__ GArgs g, const __grid_constant__ GPlane p) {
  fsl_pdl_enter();
  const GInst I = g_inst(g, blockIdx.y);
  if (!I.active) return;
  using T = greal<V>;
  extern __shared__ __align__(16) unsigned char g_smem[];
  V* twx = reinterpret_cast<V*>(g_smem);
  V* twy = twx + g.mx;
  V* pl = twy + g.my;
  V* ex = twx + p.ex_off;
  for (int i = threadIdx.x; i < g.mx; i += blockDim.x) twx[i] = reinterpret_cast<const V*>(p.twx)[i];
  for (int i = threadIdx.x; i < g.my; i += blockDim.x) twy[i] = reinterpret_cast<const V*>(p.twy)[i];
  const int mx = g.mx, my = g.my;
  const V* in = reinterpret_cast<const V*>(I.spec) + (size_t)blockIdx.x * my * g.mxh;
  __syncthreads();
  {
    const int t = threadIdx.x / p.ly, cl = threadIdx.x - t * p.ly;
    auto pos = [&](int a, int tt) { return (a * p.ay.t + tt) * p.ly + cl; };
    for (int c0 = 0; c0 < g.mxh; c0 += p.ly) {
      const int c = c0 + cl;
      const bool on = t < p.ay.t && c < g.mxh;
      if (on) gfirst<V, 1, RMAX>(p.ay, t, ex, [&](int y) { return in[(size_t)y * g.mxh + c]; }, pos);
      __syncthreads();
      if (on) gsecond<V, 1, RMAX>(p.ay, t, ex, twy, pos, [&](int y, V v) { pl[y * p.pitch + c] = v; });
      __syncthreads();
    }
  }
  {
    const int l = threadIdx.x / p.ax.t, t = threadIdx.x - l * p.ax.t;
    const T sc = (T)p.scale;
    T* out = reinterpret_cast<T*>(I.v) + (size_t)blockIdx.x * mx * my;
    const T* u = reinterpret_cast<const T*>(I.u) + (size_t)blockIdx.x * mx * my;
    auto pos = [&](int a, int tt) { return a * p.nt + l * p.ax.t + tt; };
    for (int g0 = 0; g0 < p.npairs; g0 += p.lx) {
      const int pr = g0 + l;
      const bool on = l < p.lx && pr < p.npairs, two = 2 * pr + 1 < my;
      if (on) {
        const V* e0 = pl + (2 * pr) * p.pitch;
        gfirst<V, 1, RMAX>(
            p.ax, t, ex,
            [&](int x) {
              const bool lo = x < g.mxh;
              const int k = lo ? x : mx - x;
              V e = e0[k], o = two ? e0[p.pitch + k] : gmk<V>(0, 0);
              if (!lo) {
                e.y = -e.y;
                o.y = -o.y;
              }
              return gmk<V>(e.x - o.y, e.y + o.x);  // X_2p + i X_2p+1
            },
            pos);
      }
      __syncthreads();
      if (on) {
        const size_t r0 = (size_t)(2 * pr) * mx;
        gsecond<V, 1, RMAX>(p.ax, t, ex, twx, pos, [&](int x, V v) {
          T a = v.x * sc, b = v.y * sc;
          if (g.pred) {
            a = (T)0.5 * (a + u[r0 + x]);
            if (two) b = (T)0.5 * (b + u[r0 + mx + x]);
          }
          out[r0 + x] = a;
          if (two) out[r0 + mx + x] = b;
        });
      }
      __syncthreads();
    }
  }
}

// --------------------------------------------------------- one axis a pass ---
struct GLines {
  GAxis a;
  int nl;      // lines per block
  int pitch;   // x passes: buffer pitch of a line
  const void* tw;
  double scale;
};

// x passes: where a line's points wait between the stages.  Two stages:
// (a, t) at a pitch + l T + t with pitch 1 mod 16 (8 in FP64), distinct
// banks for both stages; more: line by line.

template <class V, int RMAX, bool MULTI, int NT>
__global__ void __launch_bounds__(NT) k_g_x_fwd(const __grid_constant__ GArgs g, const __grid_constant__ GLines p, int size) {
  fsl_pdl_enter();
  const GInst I = g_inst(g, blockIdx.y);
  if (!I.active) return;
  using T = greal<V>;
  extern __shared__ __align__(16) unsigned char g_smem[];
  V* tw = reinterpret_cast<V*>(g_smem);
  V *b0 = tw + g.mx, *b1 = b0 + size;
  for (int i = threadIdx.x; i < g.mx; i += blockDim.x) tw[i] = reinterpret_cast<const V*>(p.tw)[i];
  const int mx = g.mx, l = threadIdx.x / p.a.t, t = threadIdx.x - l * p.a.t;
  const long nrows = (long)g.ncomp * g.my * g.mz, np = (nrows + 1) / 2, p0 = (long)blockIdx.x * p.nl;
  const long pr = p0 + l;
  const bool on = l < p.nl && pr < np, two = 2 * pr + 1 < nrows;
  const T* r0 = reinterpret_cast<const T*>(I.w) + 2 * pr * mx;
  __syncthreads();
  // Z in order at l (mx + 1) + f of the buffer that the last stage does not
  // read
  const int zp = mx + 1;
  V* zb = MULTI && p.a.ns % 2 ? b0 : b1;
  gline<V, -1, RMAX, MULTI>(
      p.a, t, on, b0, b1, tw, [&](int a, int tt) { return a * p.pitch + l * p.a.t + tt; },
      [&](int i) { return l * p.pitch + i; }, [&](int x) { return gmk<V>(r0[x], two ? r0[mx + x] : (T)0); },
      [&](int f, V v, V* o) { o[l * zp + f] = v; });
  __syncthreads();
  V* out = reinterpret_cast<V*>(I.spec);
  const int mxh = g.mxh;
  for (int e = threadIdx.x; e < p.nl * mxh; e += blockDim.x) {
    const int q = e / mxh, k = e - q * mxh;
    const long row = 2 * (p0 + q);
    if (row >= nrows) continue;
    const V zk = zb[q * zp + k], zm = zb[q * zp + (k ? mx - k : 0)];
    const T h = (T)0.5;
    out[(size_t)row * mxh + k] = gmk<V>(h * (zk.x + zm.x), h * (zk.y - zm.y));
    if (row + 1 < nrows) out[(size_t)(row + 1) * mxh + k] = gmk<V>(h * (zk.y + zm.y), -h * (zk.x - zm.x));
  }
}

template <class V, int RMAX, bool MULTI, int NT>
__global__ void __launch_bounds__(NT) k_g_x_inv(const __grid_constant__ GArgs g, const __grid_constant__ GLines p, int size) {
  fsl_pdl_enter();
  const GInst I = g_inst(g, blockIdx.y);
  if (!I.active) return;
  using T = greal<V>;
  extern __shared__ __align__(16) unsigned char g_smem[];
  V* tw = reinterpret_cast<V*>(g_smem);
  V *b0 = tw + g.mx, *b1 = b0 + size;
  for (int i = threadIdx.x; i < g.mx; i += blockDim.x) tw[i] = reinterpret_cast<const V*>(p.tw)[i];
  const int mx = g.mx, l = threadIdx.x / p.a.t, t = threadIdx.x - l * p.a.t;
  const long nrows = (long)g.ncomp * g.my * g.mz, np = (nrows + 1) / 2;
  const long pr = (long)blockIdx.x * p.nl + l;
  const bool on = l < p.nl && pr < np, two = 2 * pr + 1 < nrows;
  const V* e0 = reinterpret_cast<const V*>(I.spec) + 2 * pr * g.mxh;
  T* o0 = reinterpret_cast<T*>(I.v) + 2 * pr * mx;
  const T* u0 = reinterpret_cast<const T*>(I.u) + 2 * pr * mx;
  const T sc = (T)p.scale;
  __syncthreads();
  gline<V, 1, RMAX, MULTI>(
      p.a, t, on, b0, b1, tw, [&](int a, int tt) { return a * p.pitch + l * p.a.t + tt; },
      [&](int i) { return l * p.pitch + i; },
      [&](int x) {
        const bool lo = x < g.mxh;
        const int k = lo ? x : mx - x;
        V e = e0[k], o = two ? e0[g.mxh + k] : gmk<V>(0, 0);
        if (!lo) {
          e.y = -e.y;
          o.y = -o.y;
        }
        return gmk<V>(e.x - o.y, e.y + o.x);
      },
      [&](int x, V v, V*) {
        T a = v.x * sc, b = v.y * sc;
        if (g.pred) {
          a = (T)0.5 * (a + u0[x]);
          if (two) b = (T)0.5 * (b + u0[mx + x]);
        }
        o0[x] = a;
        if (two) o0[mx + x] = b;
      });
}

// Complex transform along y of the half spectrum, in place: nl columns of
// one (comp, z) per block, column fastest.
template <class V, int DIR, int RMAX, bool MULTI, int NT>
__global__ void __launch_bounds__(NT) k_g_y(const __grid_constant__ GArgs g, const __grid_constant__ GLines p, int size) {
  fsl_pdl_enter();
  const GInst I = g_inst(g, blockIdx.z);
  if (!I.active) return;
  extern __shared__ __align__(16) unsigned char g_smem[];
  V* tw = reinterpret_cast<V*>(g_smem);
  V *b0 = tw + g.my, *b1 = b0 + size;
  for (int i = threadIdx.x; i < g.my; i += blockDim.x) tw[i] = reinterpret_cast<const V*>(p.tw)[i];
  const int t = threadIdx.x / p.nl, l = threadIdx.x - t * p.nl, c = blockIdx.x * p.nl + l;
  const bool on = t < p.a.t && c < g.mxh;
  V* col = reinterpret_cast<V*>(I.spec) + (size_t)blockIdx.y * g.my * g.mxh + c;
  __syncthreads();
  gline<V, DIR, RMAX, MULTI>(
      p.a, t, on, b0, b1, tw, [&](int a, int tt) { return (a * p.a.t + tt) * p.nl + l; }, [&](int i) { return i * p.nl + l; },
      [&](int y) { return col[(size_t)y * g.mxh]; },
      [&](int f, V v, V*) { col[(size_t)f * g.mxh] = v; });
}

// z transform of all three components of kx columns of one ky, the solve of
// every mode, and back.  solve 0: Stokes, src/stokesLimitFunctions.cu:
// 2399-2451 with the shifts of src/realToComplex.cu:263-303,
//   W'_a = W_a e^{-i pi j_a/m_a};  G2 = |g|^2, g_a = 2/h_a sin(pi j_a/m_a)
//   v_a = (W'_a - g_a (g.W')/G2) / (eta G2) e^{+i pi j_a/m_a},
// zero for the zero mode; 1: the Crank-Nicolson solve with the projection,
// denominator 1 + (dt/2) eta G2 / rho (src/kernelUpdateVIncompressible.cu:
// 20-73); 2: the projection alone (src/projectionDivergenceFree.cu:21-90);
// 1 and 2 keep the zero mode.  All times 1/nc.
struct GZ {
  GAxis a;
  int kx;  // columns per block
  int solve;
  const void *tw, *sx, *sy, *sz, *ex, *ey, *ez;
};

template <class V, int RMAX, bool MULTI, int NT>
__global__ void __launch_bounds__(NT) k_g_z(const __grid_constant__ GArgs g, const __grid_constant__ GZ p, int size) {
  fsl_pdl_enter();
  const GInst I = g_inst(g, blockIdx.z);
  if (!I.active) return;
  using T = greal<V>;
  extern __shared__ __align__(16) unsigned char g_smem[];
  V* tw = reinterpret_cast<V*>(g_smem);
  V *b0 = tw + g.mz, *b1 = b0 + size;
  for (int i = threadIdx.x; i < g.mz; i += blockDim.x) tw[i] = reinterpret_cast<const V*>(p.tw)[i];
  const int NL = 3 * p.kx, t = threadIdx.x / NL, l = threadIdx.x - t * NL;
  const int comp = l / p.kx, kxl = l - comp * p.kx, kx = blockIdx.x * p.kx + kxl, ky = blockIdx.y;
  const bool on = t < p.a.t && kx < g.mxh;
  const size_t zs = (size_t)g.my * g.mxh;
  V* col = reinterpret_cast<V*>(I.spec) + (size_t)comp * g.mz * zs + (size_t)ky * g.mxh + kx;
  auto pos = [&](int a, int tt) { return (a * p.a.t + tt) * NL + l; };
  auto at = [&](int i) { return i * NL + l; };
  __syncthreads();
  gline<V, -1, RMAX, MULTI>(
      p.a, t, on, b0, b1, tw, pos, at, [&](int z) { return col[(size_t)z * zs]; }, [&](int f, V v, V* o) { o[at(f)] = v; });
  V* fb = MULTI && p.a.ns % 2 ? b0 : b1;  // the spectra in order
  V* other = fb == b0 ? b1 : b0;
  __syncthreads();
  {
    const T inv_eta = (T)(1.0 / I.eta), inv_nc = (T)1 / ((T)g.mx * (T)g.my * (T)g.mz);
    const T cn = (T)(0.5 * I.dt * I.eta / I.rho);
    const int ml = threadIdx.x % p.kx, mkx = blockIdx.x * p.kx + ml;  // blockDim.x is a multiple of kx
    const bool live = mkx < g.mxh;
    const V Ex = live ? reinterpret_cast<const V*>(p.ex)[mkx] : gmk<V>(0, 0), Ey = reinterpret_cast<const V*>(p.ey)[ky];
    const T gx = live ? (T)(2 * I.invdx) * reinterpret_cast<const T*>(p.sx)[mkx] : (T)0,
            gy = (T)(2 * I.invdy) * reinterpret_cast<const T*>(p.sy)[ky], tdz = (T)(2 * I.invdz);
    if (live)
      for (int kz = threadIdx.x / p.kx; kz < g.mz; kz += blockDim.x / p.kx) {
        V* q = fb + kz * NL + ml;
        const V E[3] = {Ex, Ey, reinterpret_cast<const V*>(p.ez)[kz]};
        const T gg[3] = {gx, gy, tdz * reinterpret_cast<const T*>(p.sz)[kz]};
        if (mkx == 0 && ky == 0 && kz == 0) {
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            const V w = q[a * p.kx];
            q[a * p.kx] = p.solve ? gmk<V>(w.x * inv_nc, w.y * inv_nc) : gmk<V>(0, 0);
          }
          continue;
        }
        V W[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const V w = q[a * p.kx];
          W[a] = gmk<V>(w.x * E[a].x + w.y * E[a].y, w.y * E[a].x - w.x * E[a].y);
        }
        const T G2 = gg[0] * gg[0] + gg[1] * gg[1] + gg[2] * gg[2], invG2 = (T)1 / G2;
        const V GW = gmk<V>(gg[0] * W[0].x + gg[1] * W[1].x + gg[2] * W[2].x, gg[0] * W[0].y + gg[1] * W[1].y + gg[2] * W[2].y);
        const T fac = p.solve == 0 ? inv_eta * invG2 * inv_nc : p.solve == 1 ? inv_nc / ((T)1 + cn * G2) : inv_nc;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const V y = gmk<V>((W[a].x - gg[a] * GW.x * invG2) * fac, (W[a].y - gg[a] * GW.y * invG2) * fac);
          q[a * p.kx] = gmk<V>(y.x * E[a].x - y.y * E[a].y, y.y * E[a].x + y.x * E[a].y);
        }
      }
  }
  __syncthreads();
  gline<V, 1, RMAX, MULTI>(
      p.a, t, on, other, fb, tw, pos, at, [&](int z) { return fb[at(z)]; }, [&](int f, V v, V*) { col[(size_t)f * zs] = v; });
}

// -------------------------------------------------------------- host side ---
// n as `want` factors of at most `cap` (no 13), largest first.
bool g_split(int n, int want, int cap, int* f) {
  if (want == 0) return n == 1;
  for (int r = std::min(cap, n); r >= 2; --r)
    if (r != 13 && n % r == 0 && g_split(n / r, want - 1, r, f + 1)) {
      f[0] = r;
      return true;
    }
  return false;
}

// Stage radices of n: the fewest factors of at most 16, and of those the
// split with the smallest largest factor (balanced stages); one stage (one
// thread a line) only for the shortest lines and primes.
bool g_radices(int n, int* f, int& ns) {
  ns = 0;
  if (n == 1) return true;
  for (ns = n <= 8 || n == 11 ? 1 : 2; ns <= kGStages; ++ns)
    for (int cap = 2; cap <= kGRad; ++cap)
      if (g_split(n, ns, cap, f)) return true;
  return false;
}

bool g_axis(int n, GAxis& a) {
  a = GAxis{};
  a.n = n;
  int f[kGStages + 1] = {};
  if (!g_radices(n, f, a.ns)) return false;
  std::copy(f, f + a.ns, a.f);
  for (int s = a.ns; s < 2; ++s) a.f[s] = 1;  // at least two stages
  a.ns = std::max(a.ns, 2);
  // threads per line: one first-stage butterfly each
  a.t = n / a.f[0];
  return true;
}

int g_rmax(const GAxis& a) {
  int m = 1;
  for (int s = 0; s < a.ns; ++s) m = std::max(m, a.f[s]);
  return m;
}

template <class V>
constexpr int g_nt(int rmax) {
  return sizeof(V) == sizeof(float2) ? 512 : rmax > 8 ? 256 : 512;
}

}  // namespace

struct GPlan {
  int f64 = 0, mx = 0, my = 0, mz = 0, mxh = 0;
  GAxis ax, ay, az;
  void* tables = nullptr;  // one allocation: twiddles, shifts and sines of each axis
  void *tw[3] = {}, *sh[3] = {}, *sn[3] = {};
  // whole planes
  bool plane = false;
  int p_rmax = 0, p_threads = 0;
  GPlane fwd, inv;
  size_t s_fwd = 0, s_inv = 0;
  // single axes
  GLines lx, ly;
  int x_threads = 0, y_threads = 0, x_size = 0, y_size = 0;
  size_t s_x = 0, s_xi = 0, s_y = 0;
  GZ z;
  int z_threads = 0, z_size = 0;
  size_t s_z = 0;
};

namespace {

// The kernel of a plan's numbers: radices of at most 8 or 16, two stages or
// more.
template <class V>
struct GK {
  using P = void (*)(GArgs, GPlane);
  using L = void (*)(GArgs, GLines, int);
  using Z = void (*)(GArgs, GZ, int);
  static P fwd(int rmax) {
    return rmax <= 8 ? (P)k_g_plane_fwd<V, 8, g_nt<V>(8)> : (P)k_g_plane_fwd<V, 16, g_nt<V>(16)>;
  }
  static P inv(int rmax) {
    return rmax <= 8 ? (P)k_g_plane_inv<V, 8, g_nt<V>(8)> : (P)k_g_plane_inv<V, 16, g_nt<V>(16)>;
  }
  static L xf(bool multi) {
    return multi ? (L)k_g_x_fwd<V, 16, true, g_nt<V>(16)> : (L)k_g_x_fwd<V, 16, false, g_nt<V>(16)>;
  }
  static L xi(bool multi) {
    return multi ? (L)k_g_x_inv<V, 16, true, g_nt<V>(16)> : (L)k_g_x_inv<V, 16, false, g_nt<V>(16)>;
  }
  static L yf(bool multi) {
    return multi ? (L)k_g_y<V, -1, 16, true, g_nt<V>(16)> : (L)k_g_y<V, -1, 16, false, g_nt<V>(16)>;
  }
  static L yi(bool multi) {
    return multi ? (L)k_g_y<V, 1, 16, true, g_nt<V>(16)> : (L)k_g_y<V, 1, 16, false, g_nt<V>(16)>;
  }
  static Z z(int rmax, bool multi) {
    return multi ? (Z)k_g_z<V, 16, true, g_nt<V>(16)>
           : rmax <= 8 ? (Z)k_g_z<V, 8, false, g_nt<V>(8)>
                       : (Z)k_g_z<V, 16, false, g_nt<V>(16)>;
  }
};

// Raises f's dynamic shared-memory limit to the most the device allows
// beside its static part; false where `need` exceeds it.
bool g_allow(const void* f, size_t need, int optin) {
  cudaFuncAttributes a;
  if (cudaFuncGetAttributes(&a, f) != cudaSuccess) return false;
  const int most = optin - (int)a.sharedSizeBytes;
  if (most <= 0 || need > (size_t)most) return false;
  return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, most) == cudaSuccess;
}

int round_to(int n, int m) { return (n + m - 1) / m * m; }

// The smallest pitch >= n that is `r` modulo m
int pitch_mod(int n, int r, int m) {
  int p = n;
  while (p % m != ((r % m) + m) % m) ++p;
  return p;
}

template <class V>
bool g_build(GPlan* g, int optin) {
  using T = greal<V>;
  const int m[3] = {g->mx, g->my, g->mz};
  const size_t all = (size_t)m[0] + m[1] + m[2];
  std::vector<V> h(2 * all + (all + 1) / 2);
  T* sines = reinterpret_cast<T*>(h.data() + 2 * all);
  if (cudaMalloc(&g->tables, sizeof(V) * h.size()) != cudaSuccess) return false;
  size_t at = 0;
  for (int a = 0; a < 3; ++a) {
    g->tw[a] = (V*)g->tables + at;
    g->sh[a] = (V*)g->tables + all + at;
    g->sn[a] = (T*)((V*)g->tables + 2 * all) + at;
    const double pi = 3.14159265358979323846;
    for (int t = 0; t < m[a]; ++t, ++at) {
      const double ang = 2.0 * pi * (double)t / (double)m[a], half = pi * (double)t / (double)m[a];
      h[at].x = (T)std::cos(ang);
      h[at].y = (T)-std::sin(ang);
      h[all + at].x = (T)std::cos(half);
      h[all + at].y = (T)std::sin(half);
      sines[at] = (T)std::sin(half);
    }
  }
  if (cudaMemcpy(g->tables, h.data(), sizeof(V) * h.size(), cudaMemcpyHostToDevice) != cudaSuccess) return false;
  const int es = (int)sizeof(V), bank = es == 8 ? 16 : 8;
  const GAxis &ax = g->ax, &ay = g->ay, &az = g->az;
  const int npairs = (g->my + 1) / 2;
  // ---- whole planes, where both extents have two stages and a plane fits:
  // that saves a pass of the spectrum through the L2 or HBM (60 x 72 x 100,
  // 300 planes: 25 us a solve).  A quasi-2D field has two planes, so two
  // blocks do the work, which is the faster way up to about 80^2 only: a step
  // by planes and by one-axis passes 40 and 48 us at 32^2, 44 and 50 at 64^2,
  // 66 and 58 at 96^2, 72 and 58 at 128^2, 89 and 64 at 144^2; the rule does
  // not tell them apart yet.
  if (ax.ns == 2 && ay.ns == 2) {
    g->p_rmax = std::max(g_rmax(ax), g_rmax(ay));
    const int cap = g_nt<V>(g->p_rmax);
    int nt = std::max(npairs * ax.t, g->mxh * ay.t);
    nt = std::max(32, std::min(cap, round_to(nt, 32)));
    GPlane p{};
    p.ax = ax;
    p.ay = ay;
    p.npairs = npairs;
    p.twx = g->tw[0];
    p.twy = g->tw[1];
    p.scale = 1.0;
    // equal groups
    const int gx = (npairs + nt / ax.t - 1) / (nt / ax.t);
    p.lx = (npairs + gx - 1) / gx;
    const int gy = (g->mxh + nt / ay.t - 1) / (nt / ay.t);
    p.ly = (g->mxh + gy - 1) / gy;
    p.nt = pitch_mod(p.lx * ax.t, 1, bank);
    const int ex = std::max(ax.f[0] * p.nt, g->my * p.ly);
    g->fwd = p;
    g->fwd.pitch = pitch_mod(g->mx, ax.t, bank);
    g->fwd.ex_off = g->mx + g->my + npairs * g->fwd.pitch;
    g->s_fwd = (size_t)es * (g->fwd.ex_off + ex);
    g->inv = p;
    g->inv.pitch = g->mxh | 1;
    g->inv.ex_off = g->mx + g->my + g->my * g->inv.pitch;
    g->s_inv = (size_t)es * (g->inv.ex_off + ex);
    g->p_threads = nt;
    g->plane = g_allow((const void*)GK<V>::fwd(g->p_rmax), g->s_fwd, optin) &&
               g_allow((const void*)GK<V>::inv(g->p_rmax), g->s_inv, optin);
  }
  // ---- single axes
  if (!g->plane) {
    const bool mx_ = ax.ns > 2, my_ = ay.ns > 2;
    const int cap = g_nt<V>(16);
    GLines& x = g->lx;
    x = GLines{};
    x.a = ax;
    x.tw = g->tw[0];
    x.scale = 1.0;
    for (x.nl = std::max(1, cap / 2 / ax.t);; x.nl = std::max(1, x.nl / 2)) {
      x.pitch = mx_ ? g->mx | 1 : pitch_mod(x.nl * ax.t, 1, bank);
      g->x_size = std::max(mx_ ? x.nl * x.pitch : ax.f[0] * x.pitch, x.nl * (g->mx + 1));
      g->s_x = (size_t)es * (g->mx + 2 * (size_t)g->x_size);
      if (x.nl == 1 || g->s_x <= 100 * 1024) break;
    }
    // the inverse and the y passes emit to global memory: one buffer where
    // there are two stages, which doubles the blocks an SM holds (256^3: y
    // 118 us a pass, inverse x 133 us with two buffers)
    g->s_xi = mx_ ? g->s_x : (size_t)es * (g->mx + (size_t)ax.f[0] * x.pitch);
    g->x_threads = round_to(x.nl * ax.t, 32);
    GLines& y = g->ly;
    y = GLines{};
    y.a = ay;
    y.tw = g->tw[1];
    for (y.nl = std::max(1, std::min(g->mxh, cap / 2 / ay.t));; y.nl = std::max(1, y.nl / 2)) {
      g->y_size = y.nl * g->my;
      g->s_y = (size_t)es * (g->my + (my_ ? 2 : 1) * (size_t)g->y_size);
      if (y.nl == 1 || g->s_y <= 100 * 1024) break;
    }
    g->y_threads = round_to(y.nl * ay.t, 32);
    if (g->x_threads > cap || g->y_threads > cap || !g_allow((const void*)GK<V>::xf(mx_), g->s_x, optin) ||
        !g_allow((const void*)GK<V>::xi(mx_), g->s_xi, optin) || !g_allow((const void*)GK<V>::yf(my_), g->s_y, optin) ||
        !g_allow((const void*)GK<V>::yi(my_), g->s_y, optin))
      return false;
  }
  // ---- z
  {
    const bool multi = az.ns > 2;
    const int rmax = multi ? 16 : g_rmax(az), cap = g_nt<V>(rmax);
    GZ& z = g->z;
    z = GZ{};
    z.a = az;
    z.tw = g->tw[2];
    z.sx = g->sn[0];
    z.sy = g->sn[1];
    z.sz = g->sn[2];
    z.ex = g->sh[0];
    z.ey = g->sh[1];
    z.ez = g->sh[2];
    for (z.kx = std::max(1, std::min(es == 8 ? 16 : 8, std::min(g->mxh, cap / (3 * az.t))));; z.kx = std::max(1, z.kx / 2)) {
      g->z_size = 3 * z.kx * g->mz;
      g->s_z = (size_t)es * (g->mz + 2 * (size_t)g->z_size);
      if (z.kx == 1 || g->s_z <= 110 * 1024) break;
    }
    g->z_threads = 3 * z.kx * az.t;
    if (g->z_threads > cap || !g_allow((const void*)GK<V>::z(rmax, multi), g->s_z, optin)) return false;
  }
  return true;
}

GArgs g_args(const Batch& B, const GPlan* g, int ncomp, int pred) {
  GArgs a{};
  a.reps = B.one ? nullptr : B.reps;
  if (B.one) a.one = g_inst_of(*B.one, g->f64, pred);
  a.mx = g->mx;
  a.my = g->my;
  a.mz = g->mz;
  a.mxh = g->mxh;
  a.ncomp = ncomp;
  a.f64 = g->f64;
  a.pred = pred;
  return a;
}

template <class V>
int g_forward(const Batch& B, const GPlan* g, int ncomp, cudaStream_t s) {
  const GArgs a = g_args(B, g, ncomp, 0);
  if (g->plane) {
    fsl_launch(GK<V>::fwd(g->p_rmax), dim3(ncomp * g->mz, B.nrep), g->p_threads, g->s_fwd, s, a, g->fwd);
    return 1;
  }
  const long np = ((long)ncomp * g->my * g->mz + 1) / 2;
  fsl_launch(GK<V>::xf(g->ax.ns > 2), dim3((unsigned)((np + g->lx.nl - 1) / g->lx.nl), B.nrep), g->x_threads, g->s_x, s, a,
             g->lx, g->x_size);
  fsl_launch(GK<V>::yf(g->ay.ns > 2), dim3((g->mxh + g->ly.nl - 1) / g->ly.nl, ncomp * g->mz, B.nrep), g->y_threads, g->s_y, s,
             a, g->ly, g->y_size);
  return 2;
}

template <class V>
int g_inverse(const Batch& B, const GPlan* g, int ncomp, int pred, double scale, cudaStream_t s) {
  const GArgs a = g_args(B, g, ncomp, pred);
  if (g->plane) {
    GPlane p = g->inv;
    p.scale = scale;
    fsl_launch(GK<V>::inv(g->p_rmax), dim3(ncomp * g->mz, B.nrep), g->p_threads, g->s_inv, s, a, p);
    return 1;
  }
  fsl_launch(GK<V>::yi(g->ay.ns > 2), dim3((g->mxh + g->ly.nl - 1) / g->ly.nl, ncomp * g->mz, B.nrep), g->y_threads, g->s_y, s,
             a, g->ly, g->y_size);
  GLines x = g->lx;
  x.scale = scale;
  const long np = ((long)ncomp * g->my * g->mz + 1) / 2;
  fsl_launch(GK<V>::xi(g->ax.ns > 2), dim3((unsigned)((np + x.nl - 1) / x.nl), B.nrep), g->x_threads, g->s_xi, s, a, x,
             g->x_size);
  return 2;
}

template <class V>
void g_zpass(const Batch& B, const GPlan* g, int solve, cudaStream_t s) {
  GZ z = g->z;
  z.solve = solve;
  const bool multi = g->az.ns > 2;
  fsl_launch(GK<V>::z(multi ? 16 : g_rmax(g->az), multi), dim3((g->mxh + z.kx - 1) / z.kx, g->my, B.nrep), g->z_threads, g->s_z,
             s, g_args(B, g, 3, 0), z, g->z_size);
}

}  // namespace

void gplan_destroy(GPlan* g) {
  if (!g) return;
  cudaFree(g->tables);
  delete g;
}

GPlan* gplan_create(const Params& P) {
  GPlan* g = new GPlan();
  g->f64 = P.prec == PREC_F64;
  g->mx = P.mx;
  g->my = P.my;
  g->mz = P.mz;
  g->mxh = P.mxh;
  // register DFT factors (idempotent)
  float2 w32[kGRad + 1][kGRad] = {};
  double2 w64[kGRad + 1][kGRad] = {};
  for (int R = 1; R <= kGRad; ++R)
    for (int j = 0; j < R; ++j) {
      const double ang = 2 * 3.14159265358979323846 * j / R;
      w64[R][j] = make_double2(std::cos(ang), -std::sin(ang));
      w32[R][j] = make_float2((float)std::cos(ang), (float)-std::sin(ang));
    }
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess || optin <= 0)
    optin = 227 * 1024;
  if (cudaMemcpyToSymbol(c_g32, w32, sizeof(w32)) != cudaSuccess || cudaMemcpyToSymbol(c_g64, w64, sizeof(w64)) != cudaSuccess ||
      !g_axis(P.mx, g->ax) || !g_axis(P.my, g->ay) || !g_axis(P.mz, g->az) ||
      !(g->f64 ? g_build<double2>(g, optin) : g_build<float2>(g, optin))) {
    cudaGetLastError();
    gplan_destroy(g);
    return nullptr;
  }
  cudaGetLastError();
  return g;
}

int launch_g_forward(const Batch& B, const GPlan* g, int ncomp, cudaStream_t s) {
  return g->f64 ? g_forward<double2>(B, g, ncomp, s) : g_forward<float2>(B, g, ncomp, s);
}
int launch_g_inverse(const Batch& B, const GPlan* g, int ncomp, int pred, double scale, cudaStream_t s) {
  return g->f64 ? g_inverse<double2>(B, g, ncomp, pred, scale, s) : g_inverse<float2>(B, g, ncomp, pred, scale, s);
}
void launch_g_z(const Batch& B, const GPlan* g, int solve, cudaStream_t s) {
  if (g->f64) g_zpass<double2>(B, g, solve, s);
  else g_zpass<float2>(B, g, solve, s);
}

}  // namespace fsl
