// wt_sipg.cu -- rhs_wave3d! (src/wave.jl:573-611): the SIPG Laplacian of
// HexSBPSAT's apply_laplacian! (restated from README.md:57-80) on axis-aligned
// affine meshes, plus the tag-7 Sommerfeld pass (src/wave.jl:453-542), and the
// RK4 stage of the system (u, ut) fused into it.
//
// Per axis and pencil of an element (s the axis scale, r an end row, n its sign):
//   L u = s^2 G G u + alpha n s^2 (G^T)_{.r} du / H - tau s^2 du / H_r - n s dGu / (2 H_r)
// with the jumps du of u and dGu of the normal derivative over each end face,
// so a pencil needs its own N values and, per end face, the neighbour's value
// and normal derivative (trace).  The two sweeps of G stay two: with G G formed once
// (half the multiply-adds, which are not what bounds the kernel) the error against
// 64-bit values grew by a third.
//
// 3 N^2 threads per element, one per (axis, pencil), with the operator as kernel
// parameters (constant bank), so that a multiply-add costs no operand load; the
// three axes' results meet in shared memory and a node pass finishes them, its
// words loaded and stored in node order.  The fused stage adds the dissipation
// increments, updates u and ut and, from the new u still on chip, writes the
// normal-derivative traces that the next stage reads, so no separate trace,
// copy or update pass over the fields is left.  The node pass's words arrive by
// cp.async under the contractions: what bounds the kernel is the latency of its
// loads (41 % of the warps resident, 3.9 TB/s).
//
// One instantiation each for the right-hand side, the stage and the traces: a stage that
// is switched off at run time costs the right-hand side up to 30 % (1.5 million nodes, FP64
// n = 4 39 -> 31 us, n = 6 28.6 -> 22.8).
//
// Measured (FP64, n = 6, 40^3 elements, one stage, B200): 290 us, 355 with dissipation
// increments, where the
// trace, right-hand-side (thread per node, operands from shared memory), copy and
// two update kernels took 1.1 ms; 4^3 elements: 4.5 us a launch in the replayed
// graph, two launches a stage instead of eleven.
#include "wt_common.cuh"
#include "wt_async.cuh"
#include "wt_launch.cuh"
#include "wt_rk.cuh"

#include <algorithm>

namespace wt {

template <int N, typename real>
struct SipgP {
  real G[N * N];
  real c0[N], cN[N];     // G[0][l] / H[l], G[N-1][l] / H[l]
  real hend;             // H_end
  long long Ne, nn;
  const real* u;         // stage input
  const real* ut;
  real* utt;             // right-hand side (no stage update)
  const real* trace;     // [(6 e + f) N^2 + p + N q] normal-axis derivative at the face nodes of u
  real* trace_out;       // the same of the value the stage writes (or of u: TRACE)
  const real* sdiag;
  const int32_t* nbr;
  const int32_t* nbrf;
  const int32_t* bdry;
  const int32_t* bslot;
  int nbf;
  const real* bnorm;
  real bv[6];
  real tau, inv_R;
  int stage;             // fused RK4 stage of u_t = ut + koU, ut_t = L u + koV
  double dt;
  int nko;               // dissipation increments per field (0, 1 or 3 fields of nn words)
  const real* koU;
  const real* koV;
  real *yU, *accU, *outU, *yV, *accV, *outV;
};

// elements per CTA: about 200 threads
template <int N>
struct SipgEp {
  static constexpr int MAX = 3 * N * N >= 128 ? 1 : 224 / (3 * N * N);
};

// what a launch does: the right-hand side, the RK4 stage, the traces of u alone
enum { SIPG_RHS = 0, SIPG_STAGE = 1, SIPG_TRACE = 2 };

template <int N, typename real, int MODE>
__global__ void __launch_bounds__(3 * N * N * SipgEp<N>::MAX, 900 / (3 * N * N * SipgEp<N>::MAX))
    k_sipg(const __grid_constant__ SipgP<N, real> P, int epb) {
  constexpr bool TRACE = MODE == SIPG_TRACE, EPI = MODE == SIPG_STAGE;
  constexpr int N2 = N * N, N3 = N * N * N, TE = 3 * N2;
  constexpr int P1 = N | 1;        // odd row pitch: x pencils without bank conflicts
  constexpr int NS = N * N * P1;   // words of one field of an element
  extern __shared__ __align__(16) unsigned char smraw[];
  const int tid = threadIdx.x, le = tid / TE, t = tid - le * TE, ax = t / N2, pq = t - ax * N2, p = pq % N, q = pq / N;
  real* su = reinterpret_cast<real*>(smraw) + (size_t)le * NS;
  real* sr = reinterpret_cast<real*>(smraw) + (size_t)(epb + 3 * le) * NS;  // the axes' results
  const long long e = (long long)blockIdx.x * epb + le;
  const bool valid = e < P.Ne;
  const long long ec = valid ? e : 0;
  // this thread's pencil: first node and stride in the padded element
  const int pb = ax == 0 ? P1 * (p + N * q) : ax == 1 ? p + P1 * N * q : p + P1 * q;
  const int ps = ax == 0 ? 1 : ax == 1 ? P1 : P1 * N;
  // nodes t, t + TE, ... of the node pass; their place in the padded element
  constexpr int NI = (N3 + TE - 1) / TE;
  auto place = [](int w) { return w + (P1 - N) * (w / N); };
  const real s = P.sdiag[3 * ec + ax];
  // the two end faces: mode 0 none, 1 interior, 2 Dirichlet, 3 Sommerfeld; the outer value and trace
  int mode[2];
  real uo[2], to[2];
  long long nu[2], nt[2];  // where the neighbour's value and trace are
  if constexpr (!TRACE) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long fi = 2 * ax + h + 6 * ec;
      const int tag = valid ? P.bdry[fi] : 8;
      const int nb = P.nbr[fi];
      const int en = ::wt::bc_elem(nb, P.Ne);
      const int fs = P.nbrf[fi];  // fn | ori << 3
      mode[h] = tag == 0 && en >= 0 ? 1 : tag >= 1 && tag <= 6 ? 2 : tag == 7 && nb < 0 ? 3 : 0;
      uo[h] = mode[h] == 2 ? P.bv[tag - 1] : (real)0;
      to[h] = 0;
      nu[h] = nt[h] = 0;
      if (mode[h] == 1) {
        int pn, qn;
        face_perm((fs >> 3) & 7, p, q, N, pn, qn);
        const int fn = fs & 7;
        nu[h] = (long long)en * N3 + face_node(faxis(fn), frow(fn, N), pn, qn, N);
        nt[h] = ((long long)6 * en + fn) * N2 + pn + N * qn;
      }
    }
  }
  dep_wait();
#pragma unroll
  for (int it = 0; it < NI; ++it) {
    const int w = t + it * TE;
    if (w < N3) cp_async_word(su + place(w), P.u + ec * N3 + w);
  }
  cp_async_commit();
  // the words of the node pass, copied now so that their loads run under the
  // contractions (each thread reads back only its own): ut, dissipation
  // increments, RK states and accumulators
  real* sw = reinterpret_cast<real*>(smraw) + (size_t)4 * epb * NS + (size_t)le * (5 + 2 * P.nko) * N3;
  const bool ld_y = P.stage == 1 || P.stage == 2, ld_acc = P.stage >= 1;
  if constexpr (EPI) {
#pragma unroll
    for (int it = 0; it < NI; ++it) {
      const int w = t + it * TE;
      if (N3 % TE != 0 && w >= N3) break;
      const long long n = ec * N3 + w;
      cp_async_word(sw + w, P.ut + n);
      if (ld_y) {
        cp_async_word(sw + N3 + w, P.yU + n);
        cp_async_word(sw + 2 * N3 + w, P.yV + n);
      }
      if (ld_acc) {
        cp_async_word(sw + 3 * N3 + w, P.accU + n);
        cp_async_word(sw + 4 * N3 + w, P.accV + n);
      }
      for (int c = 0; c < P.nko; ++c) {
        cp_async_word(sw + (5 + c) * N3 + w, P.koU + c * P.nn + n);
        cp_async_word(sw + (5 + P.nko + c) * N3 + w, P.koV + c * P.nn + n);
      }
    }
  }
  cp_async_commit();
  if constexpr (!TRACE) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (mode[h] == 1) {
        uo[h] = P.u[nu[h]];
        to[h] = P.trace[nt[h]];
      }
  }
  cp_async_wait_group<1>();  // u
  __syncthreads();
  real v[N];
  // normal derivatives at the ends of this thread's pencil of su
  auto ends = [&]() {
    real d0 = 0, d1 = 0;
#pragma unroll
    for (int l = 0; l < N; ++l) {
      const real x = su[pb + ps * l];
      d0 += P.G[l] * x;
      d1 += P.G[(N - 1) * N + l] * x;
    }
    P.trace_out[(6 * ec + 2 * ax) * N2 + pq] = s * d0;
    P.trace_out[(6 * ec + 2 * ax + 1) * N2 + pq] = s * d1;
  };
  if constexpr (TRACE) {
    if (valid) ends();
    return;
  } else {
#pragma unroll
    for (int l = 0; l < N; ++l) v[l] = su[pb + ps * l];
    real d[N];  // s G v
#pragma unroll
    for (int l = 0; l < N; ++l) {
      real acc = 0;
#pragma unroll
      for (int m = 0; m < N; ++m) acc += P.G[l * N + m] * v[m];
      d[l] = s * acc;
    }
    // jumps over the two end faces and what they add at the end nodes and along the pencil
    real w[2], endv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int md = mode[h];
      const real nh = h ? (real)1 : (real)-1, ue = h ? v[N - 1] : v[0], de = h ? d[N - 1] : d[0];
      w[h] = 0;
      endv[h] = 0;
      if (md == 1 || md == 2) {
        const real du = ue - uo[h];
        const real dGu = md == 1 ? de - to[h] : (real)0;
        w[h] = s * ((md == 1 ? (real)0.5 : (real)1) * nh * du);
        endv[h] = -P.tau * s * s / P.hend * du - (real)0.5 * nh * s / P.hend * dGu;
      } else if (md == 3) {
        const long long nb = (long long)P.nbf * N2;
        const long long bi = (long long)::wt::bc_slot(P.bslot[2 * ax + h + 6 * ec], P.nbf) * N2 + pq;
        const real nx = P.bnorm[ax * nb + bi], wFH = P.bnorm[4 * nb + bi];
        const real utv = P.ut[ec * N3 + face_node(ax, h ? N - 1 : 0, p, q, N)];
        endv[h] = -wFH * (utv + nx * de + P.inv_R * ue);
      }
    }
#pragma unroll
    for (int l = 0; l < N; ++l) {
      real acc = P.c0[l] * w[0] + P.cN[l] * w[1];
#pragma unroll
      for (int m = 0; m < N; ++m) acc += P.G[l * N + m] * d[m];
      real r = s * acc;
      if (l == 0) r += endv[0];
      if (l == N - 1) r += endv[1];
      sr[ax * NS + pb + ps * l] = r;
    }
    __syncthreads();
    if (valid) {
      cp_async_wait_own();
#pragma unroll
      for (int it = 0; it < NI; ++it) {
        const int wn = t + it * TE;
        if (N3 % TE != 0 && wn >= N3) break;
        const int at = place(wn);
        const long long n = ec * N3 + wn;
        real kV = sr[at] + sr[NS + at] + sr[2 * NS + at];
        if constexpr (!EPI) {
          P.utt[n] = kV;
          continue;
        }
        const real vin = sw[wn], uin = su[at];
        real kU = vin;
        for (int c = 0; c < P.nko; ++c) {
          kU += sw[(5 + c) * N3 + wn];
          kV += sw[(5 + P.nko + c) * N3 + wn];
        }
        const real yU = ld_y ? sw[N3 + wn] : (real)0, yV = ld_y ? sw[2 * N3 + wn] : (real)0;
        const real aU = ld_acc ? sw[3 * N3 + wn] : (real)0, aV = ld_acc ? sw[4 * N3 + wn] : (real)0;
        // FP32 too without low parts: a step depends on (u, ut) alone, nothing stays behind in the workspace
        su[at] = rk_epilogue_v<real>(P.stage, P.dt, kU, uin, yU, aU, (real)0, P.yU, P.accU, P.outU, nullptr, n, nullptr);
        rk_epilogue_v<real>(P.stage, P.dt, kV, vin, yV, aV, (real)0, P.yV, P.accV, P.outV, nullptr, n, nullptr);
      }
    }
    if constexpr (EPI) {
      __syncthreads();
      if (valid) ends();  // traces of the new u for the next stage
    }
  }
}

template <int N, typename real>
static SipgP<N, real> sipg_params(const DevMesh& m, const SipgStage& S) {
  SipgP<N, real> P;
  const std::vector<double>&G = m.ops.G, &H = m.ops.H;
  for (int i = 0; i < N; ++i) {
    for (int j = 0; j < N; ++j) P.G[i * N + j] = (real)G[i * N + j];
    P.c0[i] = (real)(G[i] / H[i]);
    P.cN[i] = (real)(G[(N - 1) * N + i] / H[i]);
  }
  P.hend = (real)H[0];
  P.Ne = m.Ne; P.nn = m.nn;
  P.u = (const real*)S.u; P.ut = (const real*)S.ut; P.utt = (real*)S.utt;
  P.trace = (const real*)S.trace; P.trace_out = (real*)S.trace_out;
  P.sdiag = (const real*)m.sdiag; P.nbr = m.nbr; P.nbrf = m.nbrf; P.bdry = m.bdry; P.bslot = m.bslot;
  P.nbf = m.nbf; P.bnorm = (const real*)m.bnorm;
  for (int f = 0; f < 6; ++f) P.bv[f] = (real)S.bvals[f];
  P.tau = (real)S.tau; P.inv_R = (real)S.inv_R;
  P.stage = S.rkU.stage; P.dt = S.rkU.dt;
  P.nko = S.nko; P.koU = (const real*)S.koU; P.koV = (const real*)S.koV;
  P.yU = (real*)S.rkU.y; P.accU = (real*)S.rkU.acc; P.outU = (real*)S.rkU.out;
  P.yV = (real*)S.rkV.y; P.accV = (real*)S.rkV.acc; P.outV = (real*)S.rkV.out;
  return P;
}

template <int N, typename real, int MODE>
static int sipg_run(const DevMesh& m, const SipgStage& S, cudaStream_t s) {
  const SipgP<N, real> P = sipg_params<N, real>(m, S);
  // fewer elements per CTA when the mesh would not give every SM a CTA
  const int epb = (int)std::max<long long>(1, std::min<long long>(SipgEp<N>::MAX, m.Ne / 148));
  const unsigned blocks = (unsigned)((m.Ne + epb - 1) / epb);
  size_t smem = (size_t)(MODE == SIPG_TRACE ? 1 : 4) * epb * N * N * (N | 1) * sizeof(real);
  if (MODE == SIPG_STAGE) smem += (size_t)(5 + 2 * P.nko) * epb * N * N * N * sizeof(real);
  if (smem > 48 * 1024 && allow_smem(k_sipg<N, real, MODE>, smem)) return -2;
  return launch_dep(k_sipg<N, real, MODE>, blocks, 3 * N * N * epb, smem, s, P, epb);
}

template <int N, typename real>
static int sipg_mode(const DevMesh& m, const SipgStage& S, bool trace_only, cudaStream_t s) {
  return trace_only    ? sipg_run<N, real, SIPG_TRACE>(m, S, s)
         : S.rkU.on    ? sipg_run<N, real, SIPG_STAGE>(m, S, s)
                       : sipg_run<N, real, SIPG_RHS>(m, S, s);
}

int launch_sipg(const DevMesh& m, const SipgStage& S, bool trace_only, cudaStream_t s) {
#define WT_SIPG_CASE(NN) \
  case NN: return m.precision == 0 ? sipg_mode<NN, double>(m, S, trace_only, s) : sipg_mode<NN, float>(m, S, trace_only, s);
  switch (m.N) {
    WT_SIPG_CASE(2) WT_SIPG_CASE(3) WT_SIPG_CASE(4) WT_SIPG_CASE(5) WT_SIPG_CASE(6) WT_SIPG_CASE(7) WT_SIPG_CASE(8)
    default: return -4;
  }
#undef WT_SIPG_CASE
}

// this file's bounds word (bounds-check build; 0 otherwise)
WT_BOUNDS_TAKE(bounds_take_sipg)

}  // namespace wt
