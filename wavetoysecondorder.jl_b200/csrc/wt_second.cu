// wt_second.cu -- second-order-in-space forms u_tt = L u on the device
// (the SIPG form: wt_sipg.cu):
//   * wave_strong_rhs_mesh! (src/wave_strong_rhs.jl:95-341): chain-rule
//     curvilinear Laplacian with Mattsson-Nordstrom SAT and BGT Sommerfeld.
//   * wave_lap_strong_conservative_mesh! (src/wave_lap_strong.jl:183-308).
#include "wt_common.cuh"

#include <algorithm>

namespace wt {

template <int N>
struct Sp {
  static constexpr int N3 = N * N * N;
  static constexpr int N2 = N * N;
  static constexpr int EPB = N3 >= 100 ? 1 : (128 / N3);
  static constexpr int T = N3 * EPB;
};

template <int N, typename real>
__device__ __forceinline__ real ctr(const real* __restrict__ f, const real* __restrict__ GT, int i, int j, int k, int d) {
  real s = 0;
  if (d == 0) {
#pragma unroll
    for (int p = 0; p < N; ++p) s += GT[p * N + i] * f[p + N * (j + N * k)];
  } else if (d == 1) {
#pragma unroll
    for (int p = 0; p < N; ++p) s += GT[p * N + j] * f[i + N * (p + N * k)];
  } else {
#pragma unroll
    for (int p = 0; p < N; ++p) s += GT[p * N + k] * f[i + N * (j + N * p)];
  }
  return s;
}

// ---------------------------------------------------------------------------
// wave_strong_rhs_element! restated on the device.  With G^{ab}, W_b of
// k_strong_coef, d_a = Dhat_a u and dd_ab = Dhat_b d_a (a <= b):
//   u_tt = sum_ab G^{ab} dd_ab + sum_b W_b d_b
// and on an axis-a face (sign s, row r): the physical normal derivative is
// s sum_b G^{ab} d_b / |n|, |n|^2 = G^{aa}, so the interior / Dirichlet SAT is
//   -(s sum_b G^{ab} d_b + tau |n| (u - u_nbr)) / H_r.
//
// Bound by memory latency and bandwidth: 11 words a node (u, nine coefficients, the
// result; the 9 inverse-Jacobian entries and their 27 derivatives, node-major, were
// 36).  3 N^2 threads per element, one per (axis, pencil), operator in the constant
// bank: first d_a and dd_aa along the own axis, then one mixed derivative each (dd_01
// along y, dd_02 and dd_12 along z) and the boundary terms of the pencil's two ends (in
// the node pass, where most warps hold nodes of all faces, they took a third of the
// instructions), then a node pass in node order.  Measured (FP64, n = 5, 28^3 elements,
// B200): 80 us (3.0 TB/s), before 255 us.  (At N = 8 a thread spills 160 bytes.)
template <int N, typename real>
struct StrongP {
  double G[N * N];
  double H[N];
  double invH;  // 1 / H_end
  long long Ne, nn;
  const real* u;
  const real* ut;
  real* utt;
  const double* sc;
  const double* detjac;
  const double* Hphys;
  const int32_t* nbr;
  const int32_t* nbrf;
  const int32_t* bdry;
  double tau, inv_R;
};

// elements per CTA: about 200 threads
template <int N>
struct Pen {
  static constexpr int EPB = 3 * N * N >= 128 ? 1 : 224 / (3 * N * N);
  static constexpr int T = 3 * N * N * EPB;
};

template <int N, typename real>
__global__ void __launch_bounds__(Pen<N>::T, (N >= 7 ? 588 : 1024) / Pen<N>::T) k_strong(const __grid_constant__ StrongP<N, real> P) {
  constexpr int N2 = N * N, N3 = N * N * N, TE = 3 * N2, EPB = Pen<N>::EPB;
  constexpr int P1 = N | 1;       // odd row pitch: x pencils without bank conflicts
  constexpr int NS = N * N * P1;  // words of one field of an element
  constexpr int NI = (N3 + TE - 1) / TE;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int tid = threadIdx.x, le = tid / TE, t = tid - le * TE, ax = t / N2, pq = t - ax * N2, p = pq % N, q = pq / N;
  double* su = reinterpret_cast<double*>(smraw) + (size_t)le * (10 * NS + 6 * N2);
  double* sd = su + NS;       // d_0, d_1, d_2
  double* sdd = su + 4 * NS;  // dd_00, dd_11, dd_22, dd_01, dd_02, dd_12
  double* suf = su + 10 * NS; // the face nodes' boundary terms
  const long long e = (long long)blockIdx.x * EPB + le;
  const bool valid = e < P.Ne;
  const long long ec = valid ? e : 0;
  auto place = [](int w) { return w + (P1 - N) * (w / N); };
#pragma unroll
  for (int it = 0; it < NI; ++it) {
    const int w = t + it * TE;
    if (w < N3) su[place(w)] = valid ? (double)P.u[ec * N3 + w] : 0.0;
  }
  double uf[2];  // the neighbours' values at the ends of this thread's pencil (0 without one)
  int tag[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int f = 2 * ax + h;
    const int en = valid ? ::wt::bc_elem(P.nbr[f + 6 * ec], P.Ne) : -1;
    tag[h] = valid ? P.bdry[f + 6 * ec] : 8;
    uf[h] = en >= 0 ? (double)P.u[(long long)en * N3 + nbr_face_node(P.nbrf[f + 6 * ec], p, q, N)] : 0.0;
  }
  __syncthreads();
  {
    const int pb = ax == 0 ? P1 * (p + N * q) : ax == 1 ? p + P1 * N * q : p + P1 * q;
    const int ps = ax == 0 ? 1 : ax == 1 ? P1 : P1 * N;
    double v[N], d[N];
#pragma unroll
    for (int l = 0; l < N; ++l) v[l] = su[pb + ps * l];
#pragma unroll
    for (int l = 0; l < N; ++l) {
      double s = 0;
#pragma unroll
      for (int m = 0; m < N; ++m) s += P.G[l * N + m] * v[m];
      d[l] = s;
      sd[ax * NS + pb + ps * l] = s;
    }
#pragma unroll
    for (int l = 0; l < N; ++l) {
      double s = 0;
#pragma unroll
      for (int m = 0; m < N; ++m) s += P.G[l * N + m] * d[m];
      sdd[ax * NS + pb + ps * l] = s;
    }
  }
  __syncthreads();
  {
    // dd_01: d_0 along y; dd_02: d_0 along z; dd_12: d_1 along z
    const int pb = ax == 0 ? p + P1 * N * q : p + P1 * q, ps = ax == 0 ? P1 : P1 * N;
    const double* src = sd + (ax == 2 ? NS : 0);
    double v[N];
#pragma unroll
    for (int l = 0; l < N; ++l) v[l] = src[pb + ps * l];
#pragma unroll
    for (int l = 0; l < N; ++l) {
      double s = 0;
#pragma unroll
      for (int m = 0; m < N; ++m) s += P.G[l * N + m] * v[m];
      sdd[(3 + ax) * NS + pb + ps * l] = s;
    }
  }
  {
    const int c0 = ax, c1 = ax == 0 ? 1 : ax == 1 ? 3 : 4, c2 = ax == 0 ? 2 : ax == 1 ? 4 : 5;  // G^{ax,0..2}
    const double f0 = ax == 0 ? 1.0 : 0.5, f1 = ax == 1 ? 1.0 : 0.5, f2 = ax == 2 ? 1.0 : 0.5;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double b = 0.0;
      if (tag[h] != 8 && tag[h] >= 0 && tag[h] <= 7) {
        const int w = face_node(ax, h ? N - 1 : 0, p, q, N), at = place(w);
        const long long n = ec * N3 + w;
        const double g0 = f0 * P.sc[c0 * P.nn + n], g1 = f1 * P.sc[c1 * P.nn + n], g2 = f2 * P.sc[c2 * P.nn + n];
        const double gd = (h ? 1.0 : -1.0) * (g0 * sd[at] + g1 * sd[NS + at] + g2 * sd[2 * NS + at]);  // |n| d_n u
        const double nrm = sqrt(ax == 0 ? g0 : ax == 1 ? g1 : g2), uv = su[at];
        if (tag[h] != 7) {
          b = -gd * P.invH - P.tau * (nrm * P.invH) * (uv - uf[h]);
        } else {
          const double hpq = P.detjac[n] * P.H[p] * P.H[q];
          b = -(hpq * nrm * ((double)P.ut[n] + P.inv_R * uv) + hpq * gd) / P.Hphys[n];
        }
      }
      suf[(2 * ax + h) * N2 + pq] = b;
    }
  }
  __syncthreads();
  if (!valid) return;
#pragma unroll
  for (int it = 0; it < NI; ++it) {
    const int w = t + it * TE;
    if (N3 % TE != 0 && w >= N3) break;
    const int at = place(w);
    const long long n = ec * N3 + w;
    double c[9];
#pragma unroll
    for (int o = 0; o < 9; ++o) c[o] = P.sc[o * P.nn + n];
    double s = c[0] * sdd[at] + c[1] * sdd[3 * NS + at] + c[2] * sdd[4 * NS + at] + c[3] * sdd[NS + at] +
               c[4] * sdd[5 * NS + at] + c[5] * sdd[2 * NS + at];
    s += c[6] * sd[at];
    s += c[7] * sd[NS + at];
    s += c[8] * sd[2 * NS + at];
    const int i = w % N, j = (w / N) % N, k = w / N2;
    if (i == 0) s += suf[j + N * k];
    if (i == N - 1) s += suf[N2 + j + N * k];
    if (j == 0) s += suf[2 * N2 + i + N * k];
    if (j == N - 1) s += suf[3 * N2 + i + N * k];
    if (k == 0) s += suf[4 * N2 + i + N * j];
    if (k == N - 1) s += suf[5 * N2 + i + N * j];
    P.utt[n] = (real)s;
  }
}

// wave_lap_strong_conservative_element! on every element (uniform h).
template <int N, typename real>
__global__ void __launch_bounds__(Sp<N>::T) k_lap_strong_cons(long long Ne, const real* __restrict__ u,
                                                             real* __restrict__ Lu, double inv_h, double tau,
                                                             const int32_t* __restrict__ nbr,
                                                             const int32_t* __restrict__ nbrf,
                                                             const double* __restrict__ G,
                                                             const double* __restrict__ H) {
  constexpr int N3 = Sp<N>::N3, N2 = Sp<N>::N2, EPB = Sp<N>::EPB;
  __shared__ double GT[N2];
  __shared__ double su[EPB][N3];
  __shared__ double sdu[EPB][3][N3];
  const int tid = threadIdx.x;
  const int le = tid / N3, t = tid - le * N3;
  const int i = t % N, j = (t / N) % N, k = t / N2;
  const long long e = (long long)blockIdx.x * EPB + le;
  const bool valid = e < Ne;
  const long long ec = valid ? e : 0;
  const long long n = ec * N3 + t;
  if (tid < N2) GT[(tid % N) * N + tid / N] = G[tid];
  const double uv = valid ? (double)u[n] : 0.0;
  su[le][t] = uv;
  __syncthreads();
  double du[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    du[c] = ctr<N>(su[le], GT, i, j, k, c) * inv_h;
    sdu[le][c][t] = du[c];
  }
  __syncthreads();
  if (!valid) return;
  double s = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) s += ctr<N>(sdu[le][c], GT, i, j, k, c);
  s *= inv_h;
  const int idx3[3] = {i, j, k};
  for (int f = 0; f < 6; ++f) {
    const int al = f >> 1, fr = frow(f, N);
    if (idx3[al] != fr) continue;
    const double fs = (f & 1) ? 1.0 : -1.0;
    const double coef_neu = -fs * inv_h / H[fr];
    const double coef_dir = -tau * inv_h / H[fr];
    const int p = al == 0 ? j : i, q = al == 2 ? j : k;
    double uf = 0.0;
    const int en = ::wt::bc_elem(nbr[f + 6 * ec], Ne);
    if (en >= 0) {
      const int fs = nbrf[f + 6 * ec];  // fn | ori << 3
      uf = (double)u[(long long)en * N3 + nbr_face_node(fs, p, q, N)];
    }
    s += coef_neu * du[al];
    s += coef_dir * (uv - uf);
  }
  Lu[n] = (real)s;
}

// Scalar wave on a prescribed 4-metric (wave_curved_rhs_element! /
// wave_curved_rhs_conservative_element!, src/wave_curved_rhs.jl:45-136 and
// 217-348) on every element of a uniform Cartesian mesh: the gradients of phi
// and phidot (centred-flux SAT on the perpendicular component of each face
// unless CONS), the six Hessian components as a second G sweep of the gradient
// of phi, the pointwise solve
//   phidd = (Gam.(phidot, dphi) - 2 g^{ti} d_i phidot - g^{ij} d_ij phi) / g^{tt}
// and, when CONS, the Mattsson-Nordstrom SAT pair on the faces.  ginv holds
// (tt,tx,ty,tz,xx,xy,xz,yy,yz,zz) and gam (t,x,y,z) per node, component
// fastest; faces without a neighbour see zero traces.  FP64 arithmetic.
template <int N, typename real, bool CONS>
__global__ void __launch_bounds__(Sp<N>::T) k_curved4(long long Ne, const real* __restrict__ u,
                                                     const real* __restrict__ ud, real* __restrict__ udd,
                                                     const real* __restrict__ ginv, const real* __restrict__ gam,
                                                     double inv_h, double tau, const int32_t* __restrict__ nbr,
                                                     const int32_t* __restrict__ nbrf, const double* __restrict__ G,
                                                     const double* __restrict__ H) {
  constexpr int N3 = Sp<N>::N3, N2 = Sp<N>::N2, EPB = Sp<N>::EPB;
  __shared__ double GT[N2];
  __shared__ double su[EPB][N3];
  __shared__ double sv[EPB][N3];
  __shared__ double sdu[EPB][3][N3];
  const int tid = threadIdx.x;
  const int le = tid / N3, t = tid - le * N3;
  const int i = t % N, j = (t / N) % N, k = t / N2;
  const long long e = (long long)blockIdx.x * EPB + le;
  const bool valid = e < Ne;
  const long long ec = valid ? e : 0;
  const long long n = ec * N3 + t;
  if (tid < N2) GT[(tid % N) * N + tid / N] = G[tid];
  const double uv = valid ? (double)u[n] : 0.0, vv = valid ? (double)ud[n] : 0.0;
  su[le][t] = uv;
  sv[le][t] = vv;
  // neighbour traces of phi and phidot at this node's faces (zero without one)
  const int idx3[3] = {i, j, k};
  double uf[6], vf[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    uf[f] = 0.0;
    vf[f] = 0.0;
    const int al = f >> 1;
    if (!valid || idx3[al] != frow(f, N)) continue;
    const int en = ::wt::bc_elem(nbr[f + 6 * ec], Ne);
    if (en < 0) continue;
    const int fs = nbrf[f + 6 * ec];  // fn | ori << 3
    const int p = al == 0 ? j : i, q = al == 2 ? j : k;
    const long long src = (long long)en * N3 + nbr_face_node(fs, p, q, N);
    uf[f] = (double)u[src];
    vf[f] = (double)ud[src];
  }
  __syncthreads();
  double du[3], dv[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    du[c] = ctr<N>(su[le], GT, i, j, k, c) * inv_h;
    dv[c] = ctr<N>(sv[le], GT, i, j, k, c) * inv_h;
  }
  if (!CONS) {
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const int al = f >> 1, fr = frow(f, N);
      if (idx3[al] != fr) continue;
      const double coef = ((f & 1) ? 1.0 : -1.0) * 0.5 * (1.0 / H[fr]) * inv_h;
      du[al] += coef * (uf[f] - uv);
      dv[al] += coef * (vf[f] - vv);
    }
  }
#pragma unroll
  for (int c = 0; c < 3; ++c) sdu[le][c][t] = du[c];
  __syncthreads();
  if (!valid) return;
  // Hessian: xx, xy, xz of d_x phi; yy, yz of d_y phi; zz of d_z phi
  const double dxx = ctr<N>(sdu[le][0], GT, i, j, k, 0) * inv_h;
  const double dxy = ctr<N>(sdu[le][0], GT, i, j, k, 1) * inv_h;
  const double dxz = ctr<N>(sdu[le][0], GT, i, j, k, 2) * inv_h;
  const double dyy = ctr<N>(sdu[le][1], GT, i, j, k, 1) * inv_h;
  const double dyz = ctr<N>(sdu[le][1], GT, i, j, k, 2) * inv_h;
  const double dzz = ctr<N>(sdu[le][2], GT, i, j, k, 2) * inv_h;
  double g[10], gm[4];
#pragma unroll
  for (int c = 0; c < 10; ++c) g[c] = (double)ginv[10 * n + c];
#pragma unroll
  for (int c = 0; c < 4; ++c) gm[c] = (double)gam[4 * n + c];
  const double gdd = gm[0] * vv + gm[1] * du[0] + gm[2] * du[1] + gm[3] * du[2];
  const double gti = g[1] * dv[0] + g[2] * dv[1] + g[3] * dv[2];
  const double gij = g[4] * dxx + g[7] * dyy + g[9] * dzz + 2 * g[5] * dxy + 2 * g[6] * dxz + 2 * g[8] * dyz;
  double s = (gdd - 2 * gti - gij) / g[0];
  if (CONS) {
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const int al = f >> 1, fr = frow(f, N);
      if (idx3[al] != fr) continue;
      const double coef_neu = -((f & 1) ? 1.0 : -1.0) * inv_h * (1.0 / H[fr]);
      const double coef_dir = -(tau * inv_h) * (1.0 / H[fr]);
      s += coef_neu * du[al];
      s += coef_dir * (uv - uf[f]);
    }
  }
  udd[n] = (real)s;
}

// Prescribed 4-metrics at the nodes (eval_curved_background!,
// src/wave_curved_rhs.jl:373-418): kind 0 Minkowski, kind 1 the gauge wave
// ds^2 = (1 - H)(-dt^2 + dx^2) + dy^2 + dz^2, H = A sin(2 pi (x - t)/d)
// (Alcubierre et al. 2004), p = (A, d).  Its inverse is diag(-1/(1-H),
// 1/(1-H), 1, 1) and its contracted Christoffels vanish (harmonic gauge).
template <typename real>
__global__ void k_curved4_bg(long long nn, const double* __restrict__ coords, int kind, double A, double d, double t,
                             real* __restrict__ ginv, real* __restrict__ gam) {
  for (long long n = blockIdx.x * (long long)blockDim.x + threadIdx.x; n < nn; n += (long long)gridDim.x * blockDim.x) {
    double f = 1.0;
    if (kind == 1) f = 1.0 - A * sin(2.0 * M_PI * (coords[3 * n] - t) / d);
    real* g = ginv + 10 * n;
#pragma unroll
    for (int c = 0; c < 10; ++c) g[c] = (real)0;
    g[0] = (real)(-1.0 / f);
    g[4] = (real)(1.0 / f);
    g[7] = (real)1;
    g[9] = (real)1;
#pragma unroll
    for (int c = 0; c < 4; ++c) gam[4 * n + c] = (real)0;
  }
}

// ---------------------------------------------------------------------------
#define WT_DISPATCH_N2(N_, CALL)  \
  switch (N_) {                   \
    case 2: { constexpr int NN = 2; return CALL; } \
    case 3: { constexpr int NN = 3; return CALL; } \
    case 4: { constexpr int NN = 4; return CALL; } \
    case 5: { constexpr int NN = 5; return CALL; } \
    case 6: { constexpr int NN = 6; return CALL; } \
    case 7: { constexpr int NN = 7; return CALL; } \
    case 8: { constexpr int NN = 8; return CALL; } \
    default: return -4;           \
  }

template <int N, typename real>
static int strong_dispatch(const DevMesh& m, const void* u, const void* ut, void* utt, double tau, double inv_R,
                           cudaStream_t s) {
  StrongP<N, real> P;
  for (int q = 0; q < N * N; ++q) P.G[q] = m.ops.G[q];
  for (int q = 0; q < N; ++q) P.H[q] = m.ops.H[q];
  P.invH = 1.0 / m.ops.H[0];
  P.Ne = m.Ne; P.nn = m.nn; P.u = (const real*)u; P.ut = (const real*)ut; P.utt = (real*)utt;
  P.sc = m.strong_c; P.detjac = m.detjac; P.Hphys = m.Hphys;
  P.nbr = m.nbr; P.nbrf = m.nbrf; P.bdry = m.bdry; P.tau = tau; P.inv_R = inv_R;
  constexpr int EPB = Pen<N>::EPB;
  const unsigned blocks = (unsigned)((m.Ne + EPB - 1) / EPB);
  const size_t smem = (size_t)EPB * (10 * N * N * (N | 1) + 6 * N * N) * sizeof(double);
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(k_strong<N, real>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
    return -2;
  k_strong<N, real><<<blocks, Pen<N>::T, smem, s>>>(P);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int launch_strong(const DevMesh& m, const void* u, const void* ut, void* utt, double tau, double inv_R,
                  cudaStream_t s) {
  if (m.precision == 0) {
    WT_DISPATCH_N2(m.N, (strong_dispatch<NN, double>(m, u, ut, utt, tau, inv_R, s)));
  } else {
    WT_DISPATCH_N2(m.N, (strong_dispatch<NN, float>(m, u, ut, utt, tau, inv_R, s)));
  }
}

template <int N, typename real>
static int lsc_dispatch(const DevMesh& m, const void* u, void* Lu, double h, double tau, cudaStream_t s) {
  const unsigned blocks = (unsigned)((m.Ne + Sp<N>::EPB - 1) / Sp<N>::EPB);
  k_lap_strong_cons<N, real><<<blocks, Sp<N>::T, 0, s>>>(m.Ne, (const real*)u, (real*)Lu, 1.0 / h, tau, m.nbr,
                                                         m.nbrf, m.G, m.H);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int launch_lap_strong_cons(const DevMesh& m, const void* u, void* Lu, double h, double tau, cudaStream_t s) {
  if (m.precision == 0) {
    WT_DISPATCH_N2(m.N, (lsc_dispatch<NN, double>(m, u, Lu, h, tau, s)));
  } else {
    WT_DISPATCH_N2(m.N, (lsc_dispatch<NN, float>(m, u, Lu, h, tau, s)));
  }
}

template <int N, typename real>
static int c4_dispatch(const DevMesh& m, const void* u, const void* ud, void* udd, const void* ginv, const void* gam,
                       double h, int cons, double tau, cudaStream_t s) {
  const unsigned blocks = (unsigned)((m.Ne + Sp<N>::EPB - 1) / Sp<N>::EPB);
  if (cons)
    k_curved4<N, real, true><<<blocks, Sp<N>::T, 0, s>>>(m.Ne, (const real*)u, (const real*)ud, (real*)udd,
                                                          (const real*)ginv, (const real*)gam, 1.0 / h, tau, m.nbr,
                                                          m.nbrf, m.G, m.H);
  else
    k_curved4<N, real, false><<<blocks, Sp<N>::T, 0, s>>>(m.Ne, (const real*)u, (const real*)ud, (real*)udd,
                                                           (const real*)ginv, (const real*)gam, 1.0 / h, tau, m.nbr,
                                                           m.nbrf, m.G, m.H);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int launch_curved4(const DevMesh& m, const void* u, const void* ud, void* udd, const void* ginv, const void* gam,
                   double h, int conservative, double tau, cudaStream_t s) {
  if (m.precision == 0) {
    WT_DISPATCH_N2(m.N, (c4_dispatch<NN, double>(m, u, ud, udd, ginv, gam, h, conservative, tau, s)));
  } else {
    WT_DISPATCH_N2(m.N, (c4_dispatch<NN, float>(m, u, ud, udd, ginv, gam, h, conservative, tau, s)));
  }
}

int launch_curved4_background(const DevMesh& m, int kind, const double* p, double t, void* ginv, void* gam,
                              cudaStream_t s) {
  const unsigned blocks = (unsigned)std::min<long long>((m.nn + 255) / 256, 8192);
  if (m.precision == 0)
    k_curved4_bg<double><<<blocks, 256, 0, s>>>(m.nn, m.coords, kind, p[0], p[1], t, (double*)ginv, (double*)gam);
  else
    k_curved4_bg<float><<<blocks, 256, 0, s>>>(m.nn, m.coords, kind, p[0], p[1], t, (float*)ginv, (float*)gam);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

// this file's bounds word (bounds-check build; 0 otherwise)
WT_BOUNDS_TAKE(bounds_take_second)

}  // namespace wt
