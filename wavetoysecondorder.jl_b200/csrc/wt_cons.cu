// wt_cons.cu -- the hot path: the conservative first-order (Phi, Pi) ADM wave
// right-hand side of wave3d_curved_rhs! (src/wave3d_curved.jl:205-258) with
// its boundary passes (src/boundaries3d.jl:58-232), Kreiss-Oliger
// dissipation (src/wave3d_curved.jl:182-192) and the RK4 stage update.
//
// One RHS evaluation is two element-parallel kernels (the two-pass structure
// HexSBPSAT uses, GOALS.md:138-151, because the divergence SAT needs the
// neighbour's flux, which needs the neighbour's gradient):
//   K1  per element: Phi -> smem, neighbour Phi face traces -> smem; split-form
//       (or affine per-axis) gradient with centred-flux SAT; flux
//       F^i = beta^i Pi + K^{ij} d_j Phi; Phidot = beta.grad + a Pi; boundary
//       increments; writes F (3 fields) and either Phidot or the fused RK4
//       stage update of Phi.
//   K2  per element: F -> smem, neighbour F face traces -> smem; split-form
//       divergence with centred-flux SAT; adds the boundary increments; writes
//       Pidot or the fused RK4 stage update of Pi.
// Every element block is a contiguous N^3 run, so all global loads are fully
// coalesced.  Streamed coefficients: a, beta (3), K (6) and, curvilinear, Ja (9)
// and 1/J.
#include "wt_common.cuh"
#include "wt_async.cuh"
#include "wt_launch.cuh"
#include "wt_rk.cuh"

#include <initializer_list>
#include <type_traits>

namespace wt {

template <int N>
struct Ep {
  static constexpr int N3 = N * N * N;
  static constexpr int N2 = N * N;
  static constexpr int EPB = N3 >= 100 ? 1 : (128 / N3);
  static constexpr int T = N3 * EPB;
};

template <typename real>
struct K1P {
  long long Ne, nn;
  long long e0, e1;  // single-solve launches: the elements [e0, e1) the launch covers
  const real* Phi;
  const real* Pi;
  const real* c10;  // a, b1, b2, b3, K11, K12, K13, K22, K23, K33 (nullptr: gradient only)
  const real* Ja;
  const real* invdetJ;
  const real* sdiag;
  const int32_t* bdry;
  const int32_t* bslot;
  const int32_t* emask;  // per element: SAT face mask (bits 0-5), outer face (bit 6)
  const int32_t* fsrc;   // per (f,e): 8 * neighbour + neighbour face, -1 without SAT
  const double* H;
  real* F;
  real* Phidot;
  real* bbuf;
  real* grad_out;
  int bc_on, bc_curv, exc_tag, nbf;
  int kinds[6];
  real sigma;
  const real* bnorm;
  const real* gPhi;
  const real* gPi;
  const real* gDx;
  const real* gDy;
  const real* gDz;
  int epi, stage;
  double dt;
  real* y;
  real* acc;
  real* out;
  real* comp;
  unsigned int* nonfinite;
  // compensated FP32 form (CP instantiation): the Phi the stage reads is Phi +
  // Phit (Phit: the state's low part at stage 0, the previous stage's small
  // output after it; NULL = zero); Ja = Ja0 [9e + c] (FP64, element constant)
  // + dJa (FP32, node order); stage 2 copies Phi into hcopy for stage 3
  const real* Phit;
  const real* dJa;
  const double* Ja0;
  real* hcopy;
  // dissipation increments of Phidot: nko fields, nn words apart
  const real* ko;
  int nko;
};

// contraction along axis d of a smem field f (N^3) with transposed G (GT[p*N+i] = G[i][p])
template <int N, typename real>
__device__ __forceinline__ real contract(const real* __restrict__ f, const real* __restrict__ GT, int i, int j, int k,
                                         int d) {
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

// the outer faces that node (i, j, k) lies on.  em: the element's emask
template <int N>
__device__ __forceinline__ int outer_faces(int em, int i, int j, int k) {
  if (!(em >> 6)) return 0;
  return ((i == 0 ? 1 : 0) | (i == N - 1 ? 2 : 0) | (j == 0 ? 4 : 0) | (j == N - 1 ? 8 : 0) | (k == 0 ? 16 : 0) |
          (k == N - 1 ? 32 : 0)) & ~em;
}

// Boundary terms of K1 at point pq = p + N q (node n) of the element's outer face f:
// the Pi part goes to the face's slot (read by K2), the Phi part is returned.  g: the
// gradient; ug: the stage's Phi; sd: the face axis's affine scale; a, b, K, Pi: the
// node's coefficients and Pi.
template <int N, typename real, typename gt>
__device__ __forceinline__ real k1_face(const K1P<real>& P, long long n, int f, int tag, int slot, int pq,
                                        const real g[3], gt ug, real sd, real Hend, real a, const real b[3],
                                        const real K[6], real Pi) {
  constexpr int N2 = Ep<N>::N2;
  const int ax = f >> 1;
  real dF = 0, dP = 0;
  if (!P.bc_curv) {
    const int kind = P.kinds[f];
    if (kind != 3) {
      const real nh = (f & 1) ? (real)1 : (real)-1;
      const real Kdd = ax == 0 ? K[0] : ax == 1 ? K[3] : K[5];
      const real a_n = sqrt(a * Kdd);
      const real bax = b[ax];
      const real bn = nh * bax;
      const real wt = sd / Hend;
      if (kind == 4) {
        const real tau = P.sigma * (fabs(a_n - bax) + fabs(a_n + bax)) * wt;
        const real gp = P.gPhi ? P.gPhi[n] : (real)0, gq = P.gPi ? P.gPi[n] : (real)0;
        dF = -tau * ((real)ug - gp);
        dP = -tau * (Pi - gq);
      } else {
        const real qv = nh * g[ax];
        const real r = Pi + ((bn + a_n) / a) * qv;
        const real gv = kind == 2 ? (real)0 : (P.gPhi ? P.gPhi[n] : (real)0);
        dP = -P.sigma * fabs(a_n + bn) * wt * (r - gv);
      }
    }
  } else if (tag != P.exc_tag) {
    const int kind = P.kinds[0];
    const long long nb = (long long)P.nbf * N2;
    const long long bi = (long long)slot * N2 + pq;
    const real nx = P.bnorm[bi], ny = P.bnorm[nb + bi], nz = P.bnorm[2 * nb + bi], wt = P.bnorm[3 * nb + bi];
    const real Kn = K[0] * nx * nx + K[3] * ny * ny + K[5] * nz * nz +
                    (real)2 * (K[1] * nx * ny + K[2] * nx * nz + K[4] * ny * nz);
    const real a_n = sqrt(a * Kn);
    const real bn = b[0] * nx + b[1] * ny + b[2] * nz;
    if (kind == 4) {
      const real tau = P.sigma * (fabs(a_n - bn) + fabs(a_n + bn)) * wt;
      const real gp = P.gPhi ? P.gPhi[n] : (real)0, gq = P.gPi ? P.gPi[n] : (real)0;
      dF = -tau * ((real)ug - gp);
      dP = -tau * (Pi - gq);
    } else {
      const real qv = nx * g[0] + ny * g[1] + nz * g[2];
      const real r = Pi + ((bn + a_n) / a) * qv;
      real gv = 0;
      if (kind != 2) {
        const real gq = P.gPi ? P.gPi[n] : (real)0;
        const real gx = P.gDx ? P.gDx[n] : (real)0, gy = P.gDy ? P.gDy[n] : (real)0,
                   gz = P.gDz ? P.gDz[n] : (real)0;
        gv = gq + ((bn + a_n) / a) * (nx * gx + ny * gy + nz * gz);
      }
      dP = -P.sigma * fabs(a_n + bn) * wt * (r - gv);
    }
  }
  P.bbuf[(long long)slot * N2 + pq] = dP;
  return dF;
}

// The node pass of K1 at node n: flux, Phidot with its boundary increments (faces,
// sdf: the outer faces it lies on and where their increments are; NULL: none) and the
// RK4 stage update or Phidot.  g: the gradient; u: the stage input (CP: its high
// part); a, b, K, Pi: the node's coefficients and Pi.
template <int N, typename real, bool CP>
__device__ __forceinline__ void k1_finish(const K1P<real>& P, long long n, int i, int j, int k, int emask,
                                          const real* sdf, const real g[3], real u, real a, const real b[3],
                                          const real K[6], real Pi, real yv, real accv, real compv) {
  constexpr int N2 = Ep<N>::N2;
  const long long nn = P.nn;
  // flux and Phidot
  const real F0 = b[0] * Pi + (K[0] * g[0] + K[1] * g[1] + K[2] * g[2]);
  const real F1 = b[1] * Pi + (K[1] * g[0] + K[3] * g[1] + K[4] * g[2]);
  const real F2 = b[2] * Pi + (K[2] * g[0] + K[4] * g[1] + K[5] * g[2]);
  real phid = b[0] * g[0] + b[1] * g[1] + b[2] * g[2] + a * Pi;
  if (sdf)
    for (int fs = outer_faces<N>(emask, i, j, k); fs; fs &= fs - 1) {
      const int f = __ffs(fs) - 1, fa = f >> 1;
      phid += sdf[f * N2 + (fa == 0 ? j : i) + N * (fa == 2 ? j : k)];
    }
  for (int c = 0; c < P.nko; ++c) phid += P.ko[c * nn + n];
  P.F[n] = F0;
  P.F[nn + n] = F1;
  P.F[2 * nn + n] = F2;
  if constexpr (CP) {
    if (P.epi)
      rk_epilogue_cp_v(P.stage, P.dt, phid, u, compv, accv, P.y, P.acc, P.out, P.comp, P.hcopy, n, P.nonfinite);
    else
      P.Phidot[n] = phid;
  } else {
    if (P.epi)
      rk_epilogue_v<real>(P.stage, P.dt, phid, u, yv, accv, compv, P.y, P.acc, P.out, P.comp, n, P.nonfinite);
    else
      P.Phidot[n] = phid;
  }
}

// ---------------------------------------------------------------------------
// The kernels of any order.  3 N^2 threads per element, one per (axis, pencil):
// a thread takes its pencil's N values into registers and applies the operator,
// kernel parameters in the constant bank, so that a multiply-add costs no operand
// load from shared memory (with a thread per node both operands came from there,
// 24 N words a node).  What bounds the kernels now is the latency of their global
// loads at the occupancy the pencils' registers leave: N = 6 FP64, 24^3 elements,
// K1 reaches 4.7 TB/s (26 words a node), K2 3.1 TB/s (14 words).  Measured, one RK4
// step (B200, FP64 / compensated FP32; thread per node -> now): N = 4, 36^3 elements
// 1184 -> 963 / 876 -> 648 us; N = 5, 28^3 1280 -> 802 / 765 -> 544; N = 6, 24^3 1336 ->
// 950 / 942 -> 579; N = 7, 20^3 1581 -> 992 / 1118 -> 545.  Fields that are read along pencils (Phi and the metric terms in
// K1, F and the metric terms in K2) arrive by cp.async in a padded layout; axis
// al's results replace its own metric terms there, pencil by pencil, and after one
// barrier a node pass sums the three axes, in node order.  Boundary terms are
// evaluated by the threads whose pencils end on an outer face, all faces at once;
// in the node pass the faces of a warp's nodes came one after another (a square root
// and a division each), 2.5 us a launch.  Measured (B200), one RK4 step with the
// terms in the node pass / by the pencil ends: N = 4, 8^3 elements FP64 52.7 -> 39.8
// us, N = 7, 4^3 57.0 -> 42.3, N = 6, 8^3 61 -> 51; FP32 N = 4, 8^3 41.3 -> 33.1;
// N = 7, 20^3 FP64 1045 -> 992, N = 5, 28^3 FP32 585 -> 544.
//
// BATCH: the CTA's elements come from a work list of (solve, element) tiles
// and each tile reads the parameter block of its solve (plist); otherwise
// element e0 + blockIdx.x * epb + le of the single solve P0.  epb: elements per CTA.
template <int N>
struct Pen {
  static constexpr int N2 = N * N, N3 = N * N * N, TE = 3 * N2;
  static constexpr int EPB = TE >= 96 ? 1 : 160 / TE;  // the most elements a CTA holds
  static constexpr int T = TE * EPB;
  static constexpr int P1 = N | 1;       // odd row pitch: x pencils without bank conflicts
  static constexpr int NS = N * N * P1;  // words of one padded field of an element
  static constexpr int NI = (N3 + TE - 1) / TE;  // nodes per thread of the node pass
  // Threads per SM the registers are sized for.  FP64 up to N = 5: 768 (72
  // registers; 576 without spills took 15-30 % longer), N = 6: 640 with the node pass's
  // words prefetched (pf1), N = 7: 600, N = 8: 448 (N = 7 at 768: 33 % slower); FP32: 1024.
  // A thread spills up to 60 bytes at most orders; at N = 7 FP64 K2 80, batches 164; the
  // affine form at N = 2 and 4 FP64 104 and 252.
  // The affine form (CURV false) at N = 2 and 4, where the node pass is most of the work,
  // waits on its loads and takes more threads: one right-hand side of 1.5 million nodes, FP64
  // N = 4 96.0 -> 83.5 us, N = 2 112 -> 93.5; FP32 N = 4 69.0 -> 67.0, N = 2 83 -> 72 (a
  // thread per node: 88.5, 102.8, 66.0, 72.2).
  template <typename real, bool CURV>
  static constexpr int occ() {
    constexpr bool F32 = sizeof(real) == 4;
    if (!CURV && (N == 2 || N == 4)) return (F32 && N == 2 ? 1536 : 1280) / T;
    return (F32 ? 1024 : N == 8 ? 448 : N == 7 ? 600 : N == 6 ? 640 : 768) / T;
  }
  // Whether K1 copies the node pass's words (coefficients, Pi, 1/J, RK words) to
  // shared memory at kernel start: it hides their latency and costs resident
  // CTAs.  24^3 elements, one step (B200): N = 6 FP64 971 us with, 1044 without;
  // N = 4, 5, 7 FP64 7-18 % slower with, FP32 0-14 %.  K2's three words always.
  template <typename real>
  static constexpr bool pf1() { return sizeof(real) == 8 && N == 6; }
  static __device__ __forceinline__ int place(int w) { return w + (P1 - N) * (w / N); }
};

// the operator: G in FP64 (CP's gradient of Phi) and in the state's type, 1 / (2 H_end)
template <int N, typename real>
struct alignas(16) OpP {  // G off a 16-byte boundary: taken in pairs its entries spill (N = 7 FP64 K1 11 % slower)
  real c2H;
  real G[N * N];
  double Gd[N * N];
};

// where a tile's element is: false if there is none
template <bool BATCH, typename KP>
__device__ __forceinline__ bool tile_element(const KP& P0, const int2* __restrict__ tiles, long long ntiles, int epb,
                                             int le, int& sid, long long& e) {
  e = (BATCH ? 0 : P0.e0) + (long long)blockIdx.x * epb + le;
  sid = 0;
  if constexpr (BATCH) {
    if (e >= ntiles) return false;
    const int2 tl = tiles[e];
    sid = tl.x;
    e = tl.y;
    return true;
  } else {
    return e < P0.e1;
  }
}

// shared words of one element in K1: Phi (CP: and its small part), the nine metric
// terms / axis results (affine: three results)
template <int N, typename real, bool CURV, bool CP>
constexpr int k1_words() {
  return Pen<N>::NS * ((CP ? 2 : 1) + (CURV ? 9 : 3)) + (Pen<N>::template pf1<real>() ? 15 * Pen<N>::N3 : 0);
}

// CP (real = float): the compensated form -- u = Phi + Phit and D u in FP64; with
// Ja = Ja0 + dJa (Ja0 element-constant, FP64) the split form is
//   0.5 D(Ja u) + 0.5 Ja D u = (Ja0 + 0.5 dJa) D u + 0.5 D(dJa u),
// and only the last contraction, of the small dJa u, runs in FP32.
template <int N, typename real, bool CURV, bool BATCH, bool CP>
__global__ void __launch_bounds__(Pen<N>::T, Pen<N>::template occ<real, CURV>())
    k_cons_k1(const __grid_constant__ K1P<real> P0, const __grid_constant__ OpP<N, real> O,
              const K1P<real>* __restrict__ plist, const int2* __restrict__ tiles, long long ntiles, int epb, int dfw) {
  using L = Pen<N>;
  using gt = typename std::conditional<CP, double, real>::type;  // precision of u and D u
  constexpr int N2 = L::N2, N3 = L::N3, TE = L::TE, NS = L::NS, P1 = L::P1;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int tid = threadIdx.x, le = tid / TE, t = tid - le * TE, ax = t / N2, pq = t - ax * N2, p = pq % N, q = pq / N;
  real* sphi = reinterpret_cast<real*>(smraw) + (size_t)le * (k1_words<N, real, CURV, CP>() + dfw);
  real* sphit = sphi + NS;               // CP
  real* sr = sphi + (CP ? 2 : 1) * NS;   // metric terms, then the axes' results
  constexpr bool PF = L::template pf1<real>();
  real* sw = sr + (CURV ? 9 : 3) * NS;   // the node pass's own words (PF)
  real* sdf = sw + (PF ? 15 * N3 : 0);   // boundary increments of Phidot [face][pq] (dfw words)
  int sid;
  long long e;
  const bool valid = tile_element<BATCH>(P0, tiles, ntiles, epb, le, sid, e);
  const K1P<real>& P = BATCH ? plist[sid] : P0;
  const long long ec = valid ? e : 0, nn = P.nn;
  const bool pf_y = P.epi && (P.stage == 1 || P.stage == 2 || (!CP && P.comp && P.stage == 3));
  const bool pf_acc = P.epi && P.stage >= 1;
  const bool pf_comp = P.epi && P.comp && (CP || P.stage == 3);
  real jh[2] = {0, 0};  // n jump / (2 H) at the two ends
  gt un[2] = {0, 0};
  int src[2] = {-1, -1}, tag[2] = {0, 0}, emask = 0;
  real m0[3] = {0, 0, 0}, sd = 0;
  if (valid) {  // what no launch of a step writes: metric terms and tables
    if constexpr (CURV) {
      const real* ja = CP ? P.dJa : P.Ja;
#pragma unroll
      for (int it = 0; it < L::NI; ++it) {
        const int w = t + it * TE;
        if (N3 % TE != 0 && w >= N3) break;
#pragma unroll
        for (int c = 0; c < 9; ++c) cp_async_word(sr + c * NS + L::place(w), ja + c * nn + ec * N3 + w);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      src[h] = ::wt::bc_src(P.fsrc[2 * ax + h + 6 * ec], P.Ne);
      tag[h] = P.bdry[2 * ax + h + 6 * ec];
    }
    emask = P.emask[ec];
  }
  dep_wait();
  if (valid) {
#pragma unroll
    for (int it = 0; it < L::NI; ++it) {
      const int w = t + it * TE;
      if (N3 % TE != 0 && w >= N3) break;
      const long long n = ec * N3 + w;
      cp_async_word(sphi + L::place(w), P.Phi + n);
      if constexpr (CP) {
        if (P.Phit) cp_async_word(sphit + L::place(w), P.Phit + n);
      }
    }
    cp_async_commit();
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (src[h] >= 0) {
        const long long nb = (long long)(src[h] >> 6) * N3 + nbr_face_node(src[h], p, q, N);
        un[h] = P.Phi[nb];
        if constexpr (CP) {
          if (P.Phit) un[h] += (gt)P.Phit[nb];
        }
      }
    if constexpr (CP && CURV) {
#pragma unroll
      for (int c = 0; c < 3; ++c) m0[c] = (real)P.Ja0[9 * ec + 3 * ax + c];
    }
    if constexpr (!CURV) sd = P.sdiag[3 * ec + ax];
    if constexpr (PF) {
#pragma unroll
      for (int it = 0; it < L::NI; ++it) {
        const int w = t + it * TE;
        if (N3 % TE != 0 && w >= N3) break;
        const long long n = ec * N3 + w;
        if constexpr (CURV) cp_async_word(sw + w, P.invdetJ + n);
        if (P.c10) {
#pragma unroll
          for (int c = 0; c < 10; ++c) cp_async_word(sw + (1 + c) * N3 + w, P.c10 + c * nn + n);
          cp_async_word(sw + 11 * N3 + w, P.Pi + n);
        }
        if (pf_y) cp_async_word(sw + 12 * N3 + w, P.y + n);
        if (pf_acc) cp_async_word(sw + 13 * N3 + w, P.acc + n);
        if (pf_comp) cp_async_word(sw + 14 * N3 + w, P.comp + n);
      }
      cp_async_commit();
    }
  }
  cp_async_wait_group<PF ? 1 : 0>();
  __syncthreads();
  if (valid) {
    const int pb = ax == 0 ? P1 * (p + N * q) : ax == 1 ? p + P1 * N * q : p + P1 * q;
    const int ps = ax == 0 ? 1 : ax == 1 ? P1 : P1 * N;
    gt u[N];
#pragma unroll
    for (int l = 0; l < N; ++l) {
      u[l] = sphi[pb + ps * l];
      if constexpr (CP) {
        if (P.Phit) u[l] += (gt)sphit[pb + ps * l];
      }
    }
    if (src[0] >= 0) jh[0] = -((real)(un[0] - u[0]) * O.c2H);
    if (src[1] >= 0) jh[1] = (real)(un[1] - u[N - 1]) * O.c2H;
    real du[N];  // D u (CP: formed in FP64, then a gradient-sized value)
#pragma unroll
    for (int l = 0; l < N; ++l) {
      gt s = 0;
#pragma unroll
      for (int m = 0; m < N; ++m) {
        if constexpr (CP) s += O.Gd[l * N + m] * u[m];
        else s += O.G[l * N + m] * u[m];
      }
      du[l] = (real)s;
    }
    if constexpr (CURV) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        real* f = sr + (3 * ax + c) * NS + pb;
        real w[N];
#pragma unroll
        for (int l = 0; l < N; ++l) w[l] = f[ps * l] * (real)u[l];
#pragma unroll
        for (int l = 0; l < N; ++l) {
          real s = 0;
#pragma unroll
          for (int k = 0; k < N; ++k) s += O.G[l * N + k] * w[k];
          const real m = f[ps * l];  // read again: held, the pencil's terms would cost resident CTAs
          real r = (real)0.5 * s + (CP ? m0[c] + (real)0.5 * m : (real)0.5 * m) * du[l];
          if (l == 0) r += (CP ? m + m0[c] : m) * jh[0];
          if (l == N - 1) r += (CP ? m + m0[c] : m) * jh[1];
          f[ps * l] = r;
        }
      }
    } else {
      real* f = sr + ax * NS + pb;
#pragma unroll
      for (int l = 0; l < N; ++l) {
        real r = sd * du[l];
        if (l == 0) r += sd * jh[0];
        if (l == N - 1) r += sd * jh[1];
        f[ps * l] = r;
      }
    }
  }
  __syncthreads();
  const bool grad_only = P.c10 == nullptr;
  // boundary terms, each thread those of its pencil's ends
  if (valid && P.bc_on && (emask >> 6) && !grad_only) {
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      const int f = 2 * ax + h, l = h ? N - 1 : 0;
      real dF = 0;
      if ((h ? tag[1] : tag[0]) != 0) {
        const int w = ax == 0 ? l + N * pq : ax == 1 ? p + N * (l + N * q) : pq + N2 * l, at = L::place(w);
        const long long n = ec * N3 + w;
        real b[3], K[6], g[3];
        const real a = P.c10[n], Pi = P.Pi[n];
#pragma unroll
        for (int c = 0; c < 3; ++c) b[c] = P.c10[(1 + c) * nn + n];
#pragma unroll
        for (int c = 0; c < 6; ++c) K[c] = P.c10[(4 + c) * nn + n];
        const real invJ = CURV ? P.invdetJ[n] : (real)1;
#pragma unroll
        for (int c = 0; c < 3; ++c)
          g[c] = CURV ? (sr[c * NS + at] + sr[(3 + c) * NS + at] + sr[(6 + c) * NS + at]) * invJ : sr[c * NS + at];
        gt ug = sphi[at];
        if constexpr (CP) {
          if (P.Phit) ug += (gt)sphit[at];
        }
        dF = k1_face<N, real>(P, n, f, h ? tag[1] : tag[0], ::wt::bc_slot(P.bslot[f + 6 * ec], P.nbf), pq, g, ug, sd,
                              (real)P.H[0], a, b, K, Pi);
      }
      if (dfw) sdf[f * N2 + pq] = dF;
    }
  }
  if (dfw) __syncthreads();
  if (!valid) return;
  cp_async_wait_own();
#pragma unroll
  for (int it = 0; it < L::NI; ++it) {
    const int w = t + it * TE;
    if (N3 % TE != 0 && w >= N3) break;
    const long long n = ec * N3 + w;
    const int at = L::place(w);
    real a = 0, b[3] = {0, 0, 0}, K[6] = {0, 0, 0, 0, 0, 0}, Pi = 0;
    if (!grad_only) {
      const real* cw = PF ? sw + N3 + w : P.c10 + n;
      const long long cs = PF ? N3 : nn;
      a = cw[0];
#pragma unroll
      for (int c = 0; c < 3; ++c) b[c] = cw[(1 + c) * cs];
#pragma unroll
      for (int c = 0; c < 6; ++c) K[c] = cw[(4 + c) * cs];
      Pi = PF ? sw[11 * N3 + w] : P.Pi[n];
    }
    const real yv = !pf_y ? (real)0 : PF ? sw[12 * N3 + w] : P.y[n];
    const real accv = !pf_acc ? (real)0 : PF ? sw[13 * N3 + w] : P.acc[n];
    const real compv = !pf_comp ? (real)0 : PF ? sw[14 * N3 + w] : P.comp[n];
    real g[3];
    if constexpr (CURV) {
      const real invJ = PF ? sw[w] : P.invdetJ[n];
#pragma unroll
      for (int c = 0; c < 3; ++c) g[c] = (sr[c * NS + at] + sr[(3 + c) * NS + at] + sr[(6 + c) * NS + at]) * invJ;
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) g[c] = sr[c * NS + at];
    }
    if (P.grad_out) {
#pragma unroll
      for (int c = 0; c < 3; ++c) P.grad_out[c * nn + n] = g[c];
    }
    if (grad_only) continue;
    const real u = sphi[at];  // CP: the high part
    k1_finish<N, real, CP>(P, n, w % N, (w / N) % N, w / N2, emask, P.bc_on && dfw ? sdf : nullptr, g, u, a, b, K, Pi, yv,
                           accv, compv);
  }
}

template <typename real>
struct K2P {
  long long Ne, nn;
  long long e0, e1;  // single-solve launches: the elements [e0, e1) the launch covers
  const real* F0;
  const real* F1;
  const real* F2;
  const real* Ja;
  const real* invdetJ;
  const real* sdiag;
  const int32_t* bdry;
  const int32_t* bslot;
  const int32_t* emask;
  const int32_t* fsrc;
  const real* bbuf;
  int bc_on, nbf;
  real* Pidot;
  int epi, stage;
  double dt;
  real* y;
  real* acc;
  real* out;
  real* comp;
  unsigned int* nonfinite;
  const real* ko;  // dissipation increments of Pidot (see K1P)
  int nko;
};

// shared words of one element in K2: F and the nine metric terms / axis results
template <int N, bool CURV>
constexpr int k2_words() {
  return Pen<N>::NS * (CURV ? 12 : 3) + 4 * Pen<N>::N3 + 6 * Pen<N>::N2;
}

template <int N, typename real, bool CURV, bool BATCH>
__global__ void __launch_bounds__(Pen<N>::T, Pen<N>::template occ<real, CURV>())
    k_cons_k2(const __grid_constant__ K2P<real> P0, const __grid_constant__ OpP<N, real> O,
              const K2P<real>* __restrict__ plist, const int2* __restrict__ tiles, long long ntiles, int epb) {
  using L = Pen<N>;
  constexpr int N2 = L::N2, N3 = L::N3, TE = L::TE, NS = L::NS, P1 = L::P1;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int tid = threadIdx.x, le = tid / TE, t = tid - le * TE, ax = t / N2, pq = t - ax * N2, p = pq % N, q = pq / N;
  real* sF = reinterpret_cast<real*>(smraw) + (size_t)le * k2_words<N, CURV>();
  real* sJ = sF + 3 * NS;  // metric terms; axis al's result replaces its first one (affine: F_al)
  int sid;
  long long e;
  const bool valid = tile_element<BATCH>(P0, tiles, ntiles, epb, le, sid, e);
  const K2P<real>& P = BATCH ? plist[sid] : P0;
  const long long ec = valid ? e : 0, nn = P.nn;
  const real* const Fp[3] = {P.F0, P.F1, P.F2};
  real* sw = sF + (CURV ? 12 : 3) * NS;  // the node pass's own words
  real* sbb = sw + 4 * N3;               // the outer faces' boundary terms [face][pq]
  const bool pf_y = P.epi && (P.stage <= 2 || P.comp);
  const bool pf_acc = P.epi && P.stage >= 1;
  const bool pf_comp = P.epi && P.comp && P.stage == 3;
  int src[2] = {-1, -1}, slot[2] = {-1, -1}, emask = 0;
  real fn[2][CURV ? 3 : 1] = {}, sd = 0;
  if (valid) {  // what no launch of a step writes: metric terms and tables
    if constexpr (CURV) {
#pragma unroll
      for (int it = 0; it < L::NI; ++it) {
        const int w = t + it * TE;
        if (N3 % TE != 0 && w >= N3) break;
#pragma unroll
        for (int c = 0; c < 9; ++c) cp_async_word(sJ + c * NS + L::place(w), P.Ja + c * nn + ec * N3 + w);
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      src[h] = ::wt::bc_src(P.fsrc[2 * ax + h + 6 * ec], P.Ne);
      if (P.bc_on && P.bdry[2 * ax + h + 6 * ec] != 0) slot[h] = ::wt::bc_slot(P.bslot[2 * ax + h + 6 * ec], P.nbf);
    }
    if (P.bc_on) emask = P.emask[ec];
  }
  dep_wait();
  if (valid) {
#pragma unroll
    for (int it = 0; it < L::NI; ++it) {
      const int w = t + it * TE;
      if (N3 % TE != 0 && w >= N3) break;
#pragma unroll
      for (int c = 0; c < 3; ++c) cp_async_word(sF + c * NS + L::place(w), Fp[c] + ec * N3 + w);
    }
    if (emask >> 6) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (slot[h] >= 0) cp_async_word(sbb + (2 * ax + h) * N2 + pq, P.bbuf + (long long)slot[h] * N2 + pq);
        else sbb[(2 * ax + h) * N2 + pq] = 0;
      }
    }
    cp_async_commit();
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (src[h] >= 0) {
        const long long nb = (long long)(src[h] >> 6) * N3 + nbr_face_node(src[h], p, q, N);
        if constexpr (CURV) {
#pragma unroll
          for (int c = 0; c < 3; ++c) fn[h][c] = Fp[c][nb];
        } else {
          fn[h][0] = (ax == 0 ? P.F0 : ax == 1 ? P.F1 : P.F2)[nb];
        }
      }
    if constexpr (!CURV) sd = P.sdiag[3 * ec + ax];
#pragma unroll
    for (int it = 0; it < L::NI; ++it) {
      const int w = t + it * TE;
      if (N3 % TE != 0 && w >= N3) break;
      const long long n = ec * N3 + w;
      if constexpr (CURV) cp_async_word(sw + w, P.invdetJ + n);
      if (pf_y) cp_async_word(sw + N3 + w, P.y + n);
      if (pf_acc) cp_async_word(sw + 2 * N3 + w, P.acc + n);
      if (pf_comp) cp_async_word(sw + 3 * N3 + w, P.comp + n);
    }
    cp_async_commit();
  }
  cp_async_wait_group<1>();
  __syncthreads();
  if (valid) {
    const int pb = ax == 0 ? P1 * (p + N * q) : ax == 1 ? p + P1 * N * q : p + P1 * q;
    const int ps = ax == 0 ? 1 : ax == 1 ? P1 : P1 * N;
    if constexpr (CURV) {
      real w[N], r[N];
      real s0 = 0, s1 = 0;  // sum_c Ja_c (F_c,nbr - F_c) at the ends
#pragma unroll
      for (int l = 0; l < N; ++l) w[l] = r[l] = 0;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const real* Fc = sF + c * NS + pb;
        const real* Jc = sJ + (3 * ax + c) * NS + pb;
        real F[N], m[N];
#pragma unroll
        for (int l = 0; l < N; ++l) {
          F[l] = Fc[ps * l];
          m[l] = Jc[ps * l];
          w[l] += m[l] * F[l];
        }
#pragma unroll
        for (int l = 0; l < N; ++l) {
          real s = 0;
#pragma unroll
          for (int k = 0; k < N; ++k) s += O.G[l * N + k] * F[k];
          r[l] += (real)0.5 * m[l] * s;
        }
        s0 += m[0] * (fn[0][c] - F[0]);
        s1 += m[N - 1] * (fn[1][c] - F[N - 1]);
      }
      if (src[0] >= 0) r[0] -= s0 * O.c2H;
      if (src[1] >= 0) r[N - 1] += s1 * O.c2H;
#pragma unroll
      for (int l = 0; l < N; ++l) {
        real s = 0;
#pragma unroll
        for (int k = 0; k < N; ++k) s += O.G[l * N + k] * w[k];
        sJ[3 * ax * NS + pb + ps * l] = r[l] + (real)0.5 * s;
      }
    } else {
      real* Fd = sF + ax * NS + pb;
      real F[N];
#pragma unroll
      for (int l = 0; l < N; ++l) F[l] = Fd[ps * l];
#pragma unroll
      for (int l = 0; l < N; ++l) {
        real s = 0;
#pragma unroll
        for (int k = 0; k < N; ++k) s += O.G[l * N + k] * F[k];
        real r = sd * s;
        if (l == 0 && src[0] >= 0) r -= sd * O.c2H * (fn[0][0] - F[0]);
        if (l == N - 1 && src[1] >= 0) r += sd * O.c2H * (fn[1][0] - F[N - 1]);
        Fd[ps * l] = r;
      }
    }
  }
  __syncthreads();
  if (!valid) return;
  cp_async_wait_own();
#pragma unroll
  for (int it = 0; it < L::NI; ++it) {
    const int w = t + it * TE;
    if (N3 % TE != 0 && w >= N3) break;
    const long long n = ec * N3 + w;
    const int at = L::place(w);
    real dv;
    if constexpr (CURV) dv = (sJ[at] + sJ[3 * NS + at] + sJ[6 * NS + at]) * sw[w];
    else dv = sF[at] + sF[NS + at] + sF[2 * NS + at];
    if (emask >> 6) {
      const int i = w % N, j = (w / N) % N, k = w / N2;
      for (int fs = outer_faces<N>(emask, i, j, k); fs; fs &= fs - 1) {
        const int f = __ffs(fs) - 1, fa = f >> 1;
        dv += sbb[f * N2 + (fa == 0 ? j : i) + N * (fa == 2 ? j : k)];
      }
    }
    for (int c = 0; c < P.nko; ++c) dv += P.ko[c * nn + n];
    if (P.epi) {
      const real yv = pf_y ? sw[N3 + w] : (real)0;
      const real accv = pf_acc ? sw[2 * N3 + w] : (real)0;
      const real compv = pf_comp ? sw[3 * N3 + w] : (real)0;
      rk_epilogue_v<real>(P.stage, P.dt, dv, yv, yv, accv, compv, P.y, P.acc, P.out, P.comp, n, P.nonfinite);
    } else {
      P.Pidot[n] = dv;
    }
  }
}

// ---------------------------------------------------------------------------
// apply_D!(Du, u, d): s_{d,e} G_d u + centred-flux SAT on interior d-faces,
// s_{d,e} = invjac[d,d] at the element's first node.
template <int N, typename real>
__global__ void __launch_bounds__(Ep<N>::T) k_apply_D(long long Ne, const real* __restrict__ u, real* __restrict__ out,
                                                     int d, const real* __restrict__ sdiag,
                                                     const int32_t* __restrict__ nbr, const int32_t* __restrict__ nbrf,
                                                     const int32_t* __restrict__ bdry, const double* __restrict__ G,
                                                     const double* __restrict__ H) {
  constexpr int N3 = Ep<N>::N3, N2 = Ep<N>::N2, EPB = Ep<N>::EPB;
  __shared__ real GT[N2];
  __shared__ real su[EPB][N3];
  const int tid = threadIdx.x;
  const int le = tid / N3, t = tid - le * N3;
  const int i = t % N, j = (t / N) % N, k = t / N2;
  const long long e = (long long)blockIdx.x * EPB + le;
  const bool valid = e < Ne;
  const long long ec = valid ? e : 0;
  const long long n = ec * N3 + t;
  if (tid < N2) GT[(tid % N) * N + tid / N] = (real)G[tid];
  const real uv = valid ? u[n] : (real)0;
  su[le][t] = uv;
  __syncthreads();
  if (!valid) return;
  const real s = sdiag[3 * ec + d];
  real r = s * contract<N>(su[le], GT, i, j, k, d);
  const int idx3[3] = {i, j, k};
  for (int f = 2 * d; f < 2 * d + 2; ++f) {
    if (idx3[d] != frow(f, N)) continue;
    if (bdry[f + 6 * ec] != 0) continue;
    const int en = ::wt::bc_elem(nbr[f + 6 * ec], Ne);
    if (en < 0) continue;
    const int p = d == 0 ? j : i, q = d == 2 ? j : k;
    const real un = u[(long long)en * N3 + nbr_face_node(nbrf[f + 6 * ec], p, q, N)];
    const real nh = (f & 1) ? (real)1 : (real)-1;
    r += nh * s / ((real)2 * (real)H[0]) * (un - uv);
  }
  out[n] = r;
}

// ---------------------------------------------------------------------------
// launchers
template <typename real>
static K1P<real> k1p_params(const DevMesh& m, const DevCoef& c, const void* Phi, const void* Pi, void* F, void* Phidot,
                            void* bbuf, void* grad_out, const ConsBC& bc, const RKStage& rk) {
  K1P<real> P;
  P.Ne = m.Ne; P.nn = m.nn; P.e0 = 0; P.e1 = m.Ne;
  P.Phi = (const real*)Phi; P.Pi = (const real*)Pi;
  P.c10 = (const real*)c.c10;
  P.Ja = (const real*)m.Ja_r; P.invdetJ = (const real*)m.invdetJ_r; P.sdiag = (const real*)m.sdiag;
  P.bdry = m.bdry; P.bslot = m.bslot;
  P.emask = m.emask; P.fsrc = m.fsrc;
  P.H = m.H;
  P.F = (real*)F; P.Phidot = (real*)Phidot; P.bbuf = (real*)bbuf; P.grad_out = (real*)grad_out;
  P.bc_on = bc.on; P.bc_curv = bc.curv; P.exc_tag = bc.exc_tag; P.nbf = m.nbf;
  for (int f = 0; f < 6; ++f) P.kinds[f] = bc.kinds[f];
  P.sigma = (real)bc.sigma; P.bnorm = (const real*)m.bnorm;
  P.gPhi = (const real*)bc.gPhi; P.gPi = (const real*)bc.gPi;
  P.gDx = (const real*)bc.gDx; P.gDy = (const real*)bc.gDy; P.gDz = (const real*)bc.gDz;
  P.epi = rk.on; P.stage = rk.stage; P.dt = rk.dt;
  P.y = (real*)rk.y; P.acc = (real*)rk.acc; P.out = (real*)rk.out; P.comp = (real*)rk.comp; P.nonfinite = rk.nonfinite;
  P.Phit = (const real*)rk.phit; P.dJa = (const real*)m.dJa; P.Ja0 = m.Ja0; P.hcopy = (real*)rk.hcopy;
  P.ko = (const real*)rk.ko; P.nko = rk.nko;
  return P;
}

// the generic K1 runs the compensated instantiation for the default FP32 form
// (not for the gradient-only launches of the energy)
static bool gen_cp(const DevMesh& m, const void* grad_out) {
  return m.precision == WT_F32 && m.fp32_form == WT_FP32_COMPENSATED && grad_out == nullptr && m.Ja0 && m.dJa;
}

template <typename real>
static K2P<real> k2p_params(const DevMesh& m, const void* F, void* Pidot, const void* bbuf, const ConsBC& bc,
                            const RKStage& rk, unsigned int* nonfinite, const void* F1, const void* F2) {
  K2P<real> P;
  P.Ne = m.Ne; P.nn = m.nn; P.e0 = 0; P.e1 = m.Ne;
  P.F0 = (const real*)F;
  P.F1 = F1 ? (const real*)F1 : (const real*)F + m.nn;
  P.F2 = F2 ? (const real*)F2 : (const real*)F + 2 * m.nn;
  P.Ja = (const real*)m.Ja_r; P.invdetJ = (const real*)m.invdetJ_r; P.sdiag = (const real*)m.sdiag;
  P.bdry = m.bdry; P.bslot = m.bslot;
  P.emask = m.emask; P.fsrc = m.fsrc;
  P.bbuf = (const real*)bbuf; P.bc_on = bc.on; P.nbf = m.nbf;
  P.Pidot = (real*)Pidot;
  P.epi = rk.on; P.stage = rk.stage; P.dt = rk.dt;
  P.y = (real*)rk.y; P.acc = (real*)rk.acc; P.out = (real*)rk.out; P.comp = (real*)rk.comp; P.nonfinite = nonfinite;
  P.ko = (const real*)rk.ko; P.nko = rk.nko;
  return P;
}

template <int N, typename real>
static OpP<N, real> op_params(const DevMesh* m) {
  OpP<N, real> O;
  const HostOps ops = m ? HostOps() : gll_operators(N);
  const HostOps& o = m ? m->ops : ops;
  for (int q = 0; q < N * N; ++q) {
    O.G[q] = (real)o.G[q];
    O.Gd[q] = o.G[q];
  }
  O.c2H = (real)(1.0 / (2.0 * o.H[0]));
  return O;
}

// Elements per CTA.  Default (variant 0): Pen<N>::EPB (affine form at N = 2: 8 of its 13,
// 5-8 % faster), fewer where the work would otherwise leave SMs without a CTA; variants 1
// and 2 (batches): half and one.  (One CTA shape gives the same bits as another.)
template <int N, bool CURV>
static int elements_per_cta(long long ne, int variant) {
  const int all = N == 2 && !CURV ? 8 : Pen<N>::EPB;
  const int most = variant == 0 ? all : variant == 1 ? (Pen<N>::EPB + 1) / 2 : 1;
  const long long fill = ne / (2 * 148);
  return (int)(fill < 1 ? 1 : fill < most ? fill : most);
}

template <typename K>
static int gen_smem(K kernel, size_t smem) {
  if (smem <= 48 * 1024) return 0;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess ? 0 : -2;
}

// whether boundary terms of K1 reach Phidot
template <typename real>
static bool k1_phi_increments(const K1P<real>& P) {
  for (int f = 0; f < 6; ++f)
    if (P.kinds[f] == 4) return true;
  return false;
}

template <int N, typename real, bool CURV, bool BATCH, bool CP>
static int k1_run(const K1P<real>& P, const OpP<N, real>& O, const void* plist, const int2* tiles, long long ne,
                  int variant, cudaStream_t s) {
  if (ne <= 0) return 0;
  const int epb = elements_per_cta<N, CURV>(ne, variant);
  // room for the boundary increments of Phidot where there can be any (full-Dirichlet faces)
  const int dfw = BATCH || (P.bc_on && k1_phi_increments(P)) ? 6 * Pen<N>::N2 : 0;
  const size_t smem = (size_t)epb * (k1_words<N, real, CURV, CP>() + dfw) * sizeof(real);
  if (gen_smem(k_cons_k1<N, real, CURV, BATCH, CP>, smem)) return -2;
  return launch_dep<!BATCH>(k_cons_k1<N, real, CURV, BATCH, CP>, (unsigned)((ne + epb - 1) / epb), Pen<N>::TE * epb, smem, s, P,
                    O, (const K1P<real>*)plist, tiles, ne, epb, dfw);
}

template <int N, typename real, bool CURV, bool BATCH>
static int k2_run(const K2P<real>& P, const OpP<N, real>& O, const void* plist, const int2* tiles, long long ne,
                  int variant, cudaStream_t s) {
  if (ne <= 0) return 0;
  const int epb = elements_per_cta<N, CURV>(ne, variant);
  const size_t smem = (size_t)epb * k2_words<N, CURV>() * sizeof(real);
  if (gen_smem(k_cons_k2<N, real, CURV, BATCH>, smem)) return -2;
  return launch_dep<!BATCH>(k_cons_k2<N, real, CURV, BATCH>, (unsigned)((ne + epb - 1) / epb), Pen<N>::TE * epb, smem, s, P, O,
                    (const K2P<real>*)plist, tiles, ne, epb);
}

template <int N, typename real>
static int k1_dispatch(const DevMesh& m, const DevCoef& c, const void* Phi, const void* Pi, void* F, void* Phidot,
                       void* bbuf, void* grad_out, int use_metric, const ConsBC& bc, const RKStage& rk,
                       cudaStream_t s, long long e0 = 0, long long e1 = -1) {
  K1P<real> P = k1p_params<real>(m, c, Phi, Pi, F, Phidot, bbuf, grad_out, bc, rk);
  P.e0 = e0;
  P.e1 = e1 < 0 ? m.Ne : e1;
  const long long ne = P.e1 - P.e0;
  const OpP<N, real> O = op_params<N, real>(&m);
  constexpr bool F32 = std::is_same<real, float>::value;
  if (F32 && gen_cp(m, grad_out))
    return use_metric ? k1_run<N, real, true, false, F32>(P, O, nullptr, nullptr, ne, 0, s)
                      : k1_run<N, real, false, false, F32>(P, O, nullptr, nullptr, ne, 0, s);
  return use_metric ? k1_run<N, real, true, false, false>(P, O, nullptr, nullptr, ne, 0, s)
                    : k1_run<N, real, false, false, false>(P, O, nullptr, nullptr, ne, 0, s);
}

template <int N, typename real>
static int k2_dispatch(const DevMesh& m, const void* F, void* Pidot, const void* bbuf, int use_metric,
                       const ConsBC& bc, const RKStage& rk, unsigned int* nonfinite, cudaStream_t s,
                       const void* F1 = nullptr, const void* F2 = nullptr, long long e0 = 0, long long e1 = -1) {
  K2P<real> P = k2p_params<real>(m, F, Pidot, bbuf, bc, rk, nonfinite, F1, F2);
  P.e0 = e0;
  P.e1 = e1 < 0 ? m.Ne : e1;
  const OpP<N, real> O = op_params<N, real>(&m);
  return use_metric ? k2_run<N, real, true, false>(P, O, nullptr, nullptr, P.e1 - P.e0, 0, s)
                    : k2_run<N, real, false, false>(P, O, nullptr, nullptr, P.e1 - P.e0, 0, s);
}

// one launch over a work list of (solve, element) tiles; variant: elements per CTA
template <int N, typename real>
static int gen_batch(int which, bool cp, int variant, const void* plist, const int2* tiles, long long ntiles,
                     cudaStream_t s) {
  static const OpP<N, real> O = op_params<N, real>(nullptr);
  constexpr bool F32 = std::is_same<real, float>::value;
  if (which == 1)
    return F32 && cp ? k1_run<N, real, true, true, F32>(K1P<real>(), O, plist, tiles, ntiles, variant, s)
                     : k1_run<N, real, true, true, false>(K1P<real>(), O, plist, tiles, ntiles, variant, s);
  return k2_run<N, real, true, true>(K2P<real>(), O, plist, tiles, ntiles, variant, s);
}

// The launch variants a batch may be given (variant 2: n = 4 and 6), and how many of them
// are different CTA shapes: n = 4 three, two or one element a CTA, n = 5 two or one; from
// n = 6 a CTA holds one element whichever is asked for.
int cons_gen_variants(int N) { return N == 4 || N == 6 ? 3 : 2; }
template <int N>
static int gen_shapes() {
  return Pen<N>::EPB == 1 ? 1 : cons_gen_variants(N) == 3 && (Pen<N>::EPB + 1) / 2 > 1 ? 3 : 2;
}

size_t cons_gen_param_size(int precision, int which) {
  if (precision == 0) return which == 1 ? sizeof(K1P<double>) : sizeof(K2P<double>);
  return which == 1 ? sizeof(K1P<float>) : sizeof(K2P<float>);
}

void cons_gen_fill_params(int which, const SolveStage& ss, unsigned* flag, void* dst) {
  const DevMesh& m = *ss.m;
  if (m.precision == 0) {
    if (which == 1)
      *(K1P<double>*)dst = k1p_params<double>(m, *ss.c, ss.Phi, ss.Pi, ss.F, nullptr, ss.bbuf, nullptr, ss.bc, ss.rkP);
    else
      *(K2P<double>*)dst = k2p_params<double>(m, ss.F, nullptr, ss.bbuf, ss.bc, ss.rkQ, flag, nullptr, nullptr);
  } else {
    if (which == 1)
      *(K1P<float>*)dst = k1p_params<float>(m, *ss.c, ss.Phi, ss.Pi, ss.F, nullptr, ss.bbuf, nullptr, ss.bc, ss.rkP);
    else
      *(K2P<float>*)dst = k2p_params<float>(m, ss.F, nullptr, ss.bbuf, ss.bc, ss.rkQ, flag, nullptr, nullptr);
  }
}

#define WT_DISPATCH_N(N_, CALL)   \
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

static inline bool a16(const void* p) { return p == nullptr || ((uintptr_t)p & 15u) == 0; }

// The pipelined n = 8 kernels stage element blocks with bulk copies, which
// need 16-byte aligned global addresses; anything else takes the generic path.
bool cons_n8_path(const DevMesh& m, const DevCoef& c, int use_metric, const ConsBC& bc, const RKStage& rkP,
                  const RKStage& rkQ, std::initializer_list<const void*> ptrs) {
  if (m.N != 8 || !use_metric || m.Ja_n8 == nullptr) return false;
  if (c.c10 == nullptr) return false;
  if (bc.on && !bc.curv) return false;
  for (const RKStage* rk : {&rkP, &rkQ})
    if (!a16(rk->y) || !a16(rk->acc) || !a16(rk->out)) return false;
  for (const void* p : ptrs)
    if (!a16(p)) return false;
  return a16(c.c10) && a16(m.invdetJ_r);
}

int cons_gen_shapes(int N) { WT_DISPATCH_N(N, (gen_shapes<NN>())); }

bool cons_gen_cp_supported(const DevMesh& m) { return gen_cp(m, nullptr); }

int launch_cons_k1(const DevMesh& m, const DevCoef& c, const void* Phi, const void* Pi, void* F, void* Phidot,
                   void* bbuf, void* grad_out, int use_metric, const ConsBC& bc, const RKStage& rk,
                   cudaStream_t s, bool n8, long long e0, long long e1) {
  if (n8 && grad_out == nullptr)
    return launch_cons_k1_n8(m, c, Phi, Pi, F, Phidot, bbuf, bc, rk, m.errflag, s, e0, e1);
  if (m.precision == 0) {
    WT_DISPATCH_N(m.N, (k1_dispatch<NN, double>(m, c, Phi, Pi, F, Phidot, bbuf, grad_out, use_metric, bc, rk, s, e0,
                                                e1)));
  } else {
    WT_DISPATCH_N(m.N, (k1_dispatch<NN, float>(m, c, Phi, Pi, F, Phidot, bbuf, grad_out, use_metric, bc, rk, s, e0,
                                               e1)));
  }
}

int launch_cons_k2(const DevMesh& m, const void* F, void* Pidot, const void* bbuf, int use_metric,
                   const ConsBC& bc, const RKStage& rk, unsigned int* nonfinite, cudaStream_t s, bool n8,
                   long long e0, long long e1) {
  if (n8) return launch_cons_k2_n8(m, F, Pidot, bbuf, bc, rk, m.errflag, s, e0, e1);
  if (m.precision == 0) {
    WT_DISPATCH_N(m.N, (k2_dispatch<NN, double>(m, F, Pidot, bbuf, use_metric, bc, rk, nonfinite, s, nullptr,
                                                nullptr, e0, e1)));
  } else {
    WT_DISPATCH_N(m.N, (k2_dispatch<NN, float>(m, F, Pidot, bbuf, use_metric, bc, rk, nonfinite, s, nullptr,
                                               nullptr, e0, e1)));
  }
}

int launch_div3d(const DevMesh& m, const void* F, void* out, cudaStream_t s) {
  // F: 3 consecutive fields
  ConsBC bc;
  RKStage rk;
  if (m.precision == 0) {
    WT_DISPATCH_N(m.N, (k2_dispatch<NN, double>(m, F, out, nullptr, 1, bc, rk, nullptr, s)));
  } else {
    WT_DISPATCH_N(m.N, (k2_dispatch<NN, float>(m, F, out, nullptr, 1, bc, rk, nullptr, s)));
  }
}

template <int N, typename real>
static int applyD_dispatch(const DevMesh& m, const void* u, void* out, int d, cudaStream_t s) {
  const unsigned blocks = (unsigned)((m.Ne + Ep<N>::EPB - 1) / Ep<N>::EPB);
  k_apply_D<N, real><<<blocks, Ep<N>::T, 0, s>>>(m.Ne, (const real*)u, (real*)out, d, (const real*)m.sdiag, m.nbr,
                                                 m.nbrf, m.bdry, m.G, m.H);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int launch_apply_D(const DevMesh& m, const void* u, void* out, int d, cudaStream_t s) {
  if (m.precision == 0) {
    WT_DISPATCH_N(m.N, (applyD_dispatch<NN, double>(m, u, out, d, s)));
  } else {
    WT_DISPATCH_N(m.N, (applyD_dispatch<NN, float>(m, u, out, d, s)));
  }
}

int launch_cons_gen_batch(int which, int N, int precision, int epb_variant, int cp, const void* plist, const int2* tiles,
                          long long ntiles, cudaStream_t s) {
  if (precision == 0) {
    WT_DISPATCH_N(N, (gen_batch<NN, double>(which, false, epb_variant, plist, tiles, ntiles, s)));
  } else {
    WT_DISPATCH_N(N, (gen_batch<NN, float>(which, cp != 0, epb_variant, plist, tiles, ntiles, s)));
  }
}

// this file's bounds word (bounds-check build; 0 otherwise)
WT_BOUNDS_TAKE(bounds_take_cons)

}  // namespace wt
