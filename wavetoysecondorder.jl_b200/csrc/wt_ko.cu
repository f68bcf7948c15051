// wt_ko.cu -- Kreiss-Oliger dissipation eps mu^-5 sum_d D_d^6 of up to two
// fields (src/wave3d_curved.jl:182-192) along whole grid lines.
//
// D_d (apply_D!) couples only the nodes of one axis-d grid line
// (METHODS.md:151-155), so a thread keeps one pencil of one element (N values)
// in registers and the threads of a CTA hold whole element lines: applying D_d
// six times needs, per pass, only the two end values of the pencils next to it.
//
// What bounds it: per axis and field 3 words of DRAM traffic per node (the field in,
// the destination in and out) against 6 N multiply-adds.  The operator is kernel
// parameters (constant bank: no shared-memory operand loads), of which half the rows
// suffice: G is antisymmetric about its centre, G[N-1-i][N-1-p] = -G[i][p], exactly as
// stored, so an entry serves both mirrored rows (with all rows as operands the 64
// registers spill and n = 8 takes four times as long).  Only the end values go through
// shared memory, double buffered, one barrier per pass.  Axis 0 pencils are contiguous
// in memory: each warp transposes its 32 pencils through a padded shared buffer of its
// own; along axes 1 and 2 consecutive threads hold consecutive nodes and load directly.
//
// Rounding.  Sums and differences of mirrored values would halve the multiply-adds,
// but their own rounding, amplified by six passes, is 1.3 to 4.7 times the plain sums'
// error on a field that oscillates within an element (n = 8, one wavelength an element,
// FP64: 3.3e-14 -> 1.5e-13; white noise 2.4e-16 -> 3.1e-16), so the passes take the plain
// sums.  Where a pencil varies by less than half its size (at four of its nodes: all
// decide alike), the first pass takes the values relative to the pencil's centre (G's
// rows sum to zero), a difference that then hardly rounds: the error of a resolved field
// falls (pulses of width 0.1 on 24 elements, n = 8: FP64 0.62, FP32 0.06 of the plain
// sums'), and no other field's grows (within 3 %; at n = 5 and 7 by up to a third against
// a reference that counts the stored rows' sums, 1e-15, as the operator's).
//
// Measured (FP64, three axes of one field, B200): 24^3 elements of n = 8, 109 us, 40^3 of
// n = 6, 263 us (in sums and differences 97 and 250).  With the whole pencils through
// shared memory on every pass, two barriers each and the matrix read from there: 315 and
// 680 us.
#include "wt_common.cuh"
#include "wt_launch.cuh"

#include <algorithm>
#include <type_traits>
#include <vector>

namespace wt {

template <int N, typename real>
struct KoP {
  real G[(N + 1) / 2 * N];  // the upper half's rows
  const real* f[2];
  real* out[2];
  long long ostride;  // words between the outputs of consecutive axes (0: one output)
  int rmw;            // 1: out += koT D^6 f, 0: out = koT D^6 f
  real koT, cH;       // cH = 1 / (2 H_end)
  const real* sdiag;
  int nax;
  struct Axis {
    int d, len, closed, pb;  // axis, elements per line, periodic, pencils per CTA
    int parts;               // CTAs per line, N^2 / pb
    unsigned pb_magic;       // floor(2^32 / pb) + 1: __umulhi(t, magic) = t / pb for t < 1024
    unsigned b0;             // first CTA of the axis
    const int32_t* lines;
  } ax[3];
};

// CTA: pb pencils of one element line of field blockIdx.y, thread (pencil, element)
// with the pencil fastest.  (Both fields in one thread shared indices, scales and
// barriers, 28 % fewer instructions, but the registers halved the resident warps:
// 3 % slower at 40^3 n = 6, 13 % on a 4^3 step.)
template <int N, typename real, int TMAX>
__global__ void __launch_bounds__(TMAX, 1024 / TMAX) k_ko(const __grid_constant__ KoP<N, real> P) {
  constexpr int N2 = N * N, N3 = N * N * N, HH = N / 2;
  constexpr int NP = N | 1;  // odd pitch of a staged pencil: no bank conflicts
  extern __shared__ __align__(16) unsigned char smraw[];
  real* ends = reinterpret_cast<real*>(smraw);  // [2 buffers][low, high end][thread]
  const int T = blockDim.x;
  const int tid = threadIdx.x, lane = tid & 31;
  real* stage = ends + 4 * T + (tid >> 5) * 32 * NP;  // this warp's staged pencils (axis 0)
  int d = P.ax[0].d, len = P.ax[0].len, closed = P.ax[0].closed, PB = P.ax[0].pb, parts = P.ax[0].parts, a = 0;
  unsigned b0 = P.ax[0].b0, pbm = P.ax[0].pb_magic;
  const int32_t* lines = P.ax[0].lines;
#pragma unroll
  for (int q = 1; q < 3; ++q)
    if (q < P.nax && blockIdx.x >= P.ax[q].b0) {
      d = P.ax[q].d; len = P.ax[q].len; closed = P.ax[q].closed; PB = P.ax[q].pb; parts = P.ax[q].parts;
      b0 = P.ax[q].b0; pbm = P.ax[q].pb_magic; lines = P.ax[q].lines; a = q;
    }
  const unsigned blk = blockIdx.x - b0;
  const int line = blk / parts, part = blk - line * parts;
  const int sg = __umulhi(tid, pbm), pb = tid - sg * PB;  // tid / PB, tid % PB
  const bool act = sg < len;
  long long base = -1;
  real s = 0;
  if (act) {
    const int e = lines[(long long)line * len + sg];
    s = P.sdiag[3 * (long long)e + d];
    const int pp = part * PB + pb;  // the pencil, its first tangential index fastest
    base = (long long)e * N3 + (d == 0 ? N * pp : d == 1 ? pp % N + N2 * (pp / N) : pp);
  }
  dep_wait();
  const real* const fp = blockIdx.y ? P.f[1] : P.f[0];
  real* const op = (blockIdx.y ? P.out[1] : P.out[0]) + a * P.ostride;
  real v[N];
  auto load = [&](auto st) {
    constexpr int stride = decltype(st)::value;
    const real* f = fp + (act ? base : 0);
#pragma unroll
    for (int l = 0; l < N; ++l) v[l] = act ? f[l * stride] : (real)0;
  };
  if (d == 0) {
#pragma unroll
    for (int it = 0; it < N; ++it) {
      const int w = it * 32 + lane, pr = w / N;
      const long long bs = __shfl_sync(0xffffffffu, base, pr);
      v[it] = bs >= 0 ? fp[bs + w % N] : (real)0;
    }
#pragma unroll
    for (int it = 0; it < N; ++it) {
      const int w = it * 32 + lane, pr = w / N;
      stage[pr * NP + w % N] = v[it];
    }
    __syncwarp();
#pragma unroll
    for (int l = 0; l < N; ++l) v[l] = stage[lane * NP + l];
    __syncwarp();
  } else if (d == 1) {
    load(std::integral_constant<int, N>());
  } else {
    load(std::integral_constant<int, N2>());
  }
  const bool has_prev = act && (closed || sg > 0), has_next = act && (closed || sg < len - 1);
  const int tp = pb + PB * (sg == 0 ? len - 1 : sg - 1), tn = pb + PB * (sg == len - 1 ? 0 : sg + 1);
  // the centre that the first pass takes the pencil relative to, or 0 (see above):
  // magnitudes by their leading bits, half of one a step of the exponent
  auto mag = [](real a) {
    if constexpr (sizeof(real) == 8) return __double2hiint(a) & 0x7fffffff;
    else return __float_as_int(a) & 0x7fffffff;
  };
  constexpr int HALF = sizeof(real) == 8 ? 1 << 20 : 1 << 23;
  real c = v[HH];
  int mv = 0, mc = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int l = q == 0 ? 0 : q == 1 ? (N > 2 ? 2 : 1) : q == 2 ? (N > 3 ? N - 3 : 0) : N - 1;
    mv = max(mv, mag(v[l]));
    mc = max(mc, mag(v[l] - c));
  }
  if (mc >= mv - HALF) c = 0;
  // v <- D v; the sums over x, the jumps to the neighbours' ends over v
  auto pass = [&](int it, auto x) {
    real* eb = ends + (it & 1) * 2 * T;
    eb[tid] = v[0];
    eb[T + tid] = v[N - 1];
    __syncthreads();
    // the centred-flux SAT of the two end nodes
    const real lo = has_prev ? v[0] - eb[T + tp] : (real)0;
    const real hi = has_next ? eb[tn] - v[N - 1] : (real)0;
    real w[N];
#pragma unroll
    for (int p = 0; p < N; ++p) {
      const real xp = x(p), xm = x(N - 1 - p);
#pragma unroll
      for (int i = 0; i < HH; ++i) {
        const real g = P.G[i * N + p];
        w[i] = p ? w[i] + g * xp : g * xp;
        w[N - 1 - i] = p ? w[N - 1 - i] - g * xm : -(g * xm);
      }
      if (N & 1) w[HH] = p ? w[HH] + P.G[HH * N + p] * xp : P.G[HH * N] * xp;
    }
    w[0] += P.cH * lo;
    w[N - 1] += P.cH * hi;
#pragma unroll
    for (int l = 0; l < N; ++l) v[l] = s * w[l];
  };
  pass(0, [&](int p) { return v[p] - c; });
  constexpr int UN = N == 6 ? 1 : 5;  // (unrolled: 40^3 of n = 6 8 % slower, 24^3 of n = 8 4 % faster)
#pragma unroll UN
  for (int it = 1; it < 6; ++it) pass(it, [&](int p) { return v[p]; });
#pragma unroll
  for (int l = 0; l < N; ++l) v[l] *= P.koT;
  auto store = [&](auto st) {
    constexpr int stride = decltype(st)::value;
    if (!act) return;
    real* o = op + base;
    if (P.rmw) {
#pragma unroll
      for (int l = 0; l < N; ++l) v[l] += o[l * stride];
    }
#pragma unroll
    for (int l = 0; l < N; ++l) o[l * stride] = v[l];
  };
  if (d == 0) {
#pragma unroll
    for (int l = 0; l < N; ++l) stage[lane * NP + l] = v[l];
    __syncwarp();
    long long at[N];
#pragma unroll
    for (int it = 0; it < N; ++it) {
      const int w = it * 32 + lane, pr = w / N;
      const long long bs = __shfl_sync(0xffffffffu, base, pr);
      at[it] = bs >= 0 ? bs + w % N : -1;
      v[it] = stage[pr * NP + w % N];
      if (P.rmw && at[it] >= 0) v[it] += op[at[it]];
    }
#pragma unroll
    for (int it = 0; it < N; ++it)
      if (at[it] >= 0) op[at[it]] = v[it];
    __syncwarp();
  } else if (d == 1) {
    store(std::integral_constant<int, N>());
  } else {
    store(std::integral_constant<int, N2>());
  }
}

template <int N, typename real, int TMAX>
static int ko_run(const KoP<N, real>& P, unsigned blocks, int nf, int threads, cudaStream_t s) {
  const size_t smem = (size_t)threads * (4 + (N | 1)) * sizeof(real);
  if (smem > 48 * 1024) {
    // set on every launch that needs it: the attribute belongs to the current device
    if (cudaFuncSetAttribute(k_ko<N, real, TMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
      return -2;
  }
  return launch_dep(k_ko<N, real, TMAX>, dim3(blocks, nf), threads, smem, s, P);
}

template <int N, typename real>
static int ko_lines_n(const DevMesh& m, const int* axes, int nax, int nf, void* const* out, long long ostride, int rmw,
                      const void* const* f, double koT, cudaStream_t s) {
  KoP<N, real> P;
  for (int q = 0; q < (N + 1) / 2 * N; ++q) P.G[q] = (real)m.ops.G[q];
  for (int q = 0; q < 2; ++q) {
    P.f[q] = (const real*)f[q < nf ? q : 0];
    P.out[q] = (real*)out[q < nf ? q : 0];
  }
  P.ostride = ostride;
  P.rmw = rmw;
  P.koT = (real)koT;
  P.cH = (real)(1.0 / (2.0 * m.ops.H[0]));
  P.sdiag = (const real*)m.sdiag;
  P.nax = nax;
  unsigned blocks = 0;
  int threads = 32;
  for (int q = 0; q < nax; ++q) {
    const int d = axes[q], len = m.line_len[d];
    // pencils per CTA: the most (a divisor of N times N) that keeps a CTA at
    // 256 threads or fewer (512: 3 % slower at 40^3 n = 6); longer lines keep the N
    // pencils of one plane
    int g = N;
    while (g > 1 && (N % g != 0 || len * N * g > 256)) --g;
    auto& A = P.ax[q];
    A.d = d; A.len = len; A.closed = m.line_closed[d]; A.pb = N * g; A.parts = N / g;
    A.pb_magic = (unsigned)(0x100000000ull / (unsigned)A.pb) + 1u; A.b0 = blocks; A.lines = m.lines[d];
    blocks += (unsigned)m.nlines[d] * (unsigned)(N / g);
    threads = std::max(threads, (len * N * g + 31) / 32 * 32);
  }
  for (int q = nax; q < 3; ++q) P.ax[q] = P.ax[0];
  if (blocks == 0 || nf == 0) return 0;
  return threads <= 256   ? ko_run<N, real, 256>(P, blocks, nf, threads, s)
         : threads <= 512 ? ko_run<N, real, 512>(P, blocks, nf, threads, s)
                          : ko_run<N, real, 1024>(P, blocks, nf, threads, s);
}

static int ko_lines(const DevMesh& m, const int* axes, int nax, int nf, void* const* out, long long ostride, int rmw,
                    const void* const* f, double koT, cudaStream_t s) {
#define WT_KO_CASE(NN)                                                                                    \
  case NN:                                                                                                \
    return m.precision == 0 ? ko_lines_n<NN, double>(m, axes, nax, nf, out, ostride, rmw, f, koT, s)      \
                            : ko_lines_n<NN, float>(m, axes, nax, nf, out, ostride, rmw, f, koT, s);
  switch (m.N) {
    WT_KO_CASE(2) WT_KO_CASE(3) WT_KO_CASE(4) WT_KO_CASE(5) WT_KO_CASE(6) WT_KO_CASE(7) WT_KO_CASE(8)
    default: return -4;
  }
#undef WT_KO_CASE
}

// Axes whose elements form straight lines short enough for one CTA run line-
// locally; the others (multi-patch meshes, whose axis-d neighbours may meet at
// another face or orientation) as the reference's _ko_axis3! does it
// (src/wave3d_curved.jl:182-192): six apply_D! calls ping-ponging through scratch
// (2 nn words), then dst += koT * result.
static bool ko_axis_lines(const DevMesh& m, int d) { return m.line_ok[d] && m.line_len[d] * m.N <= 1024; }

bool ko_all_lines(const DevMesh& m) { return ko_axis_lines(m, 0) && ko_axis_lines(m, 1) && ko_axis_lines(m, 2); }

int launch_ko_add(const DevMesh& m, int nf, void* const* dst, const void* const* field, double koT, cudaStream_t s,
                  void* scratch, int* launches) {
  for (int d = 0; d < 3; ++d) {
    if (ko_axis_lines(m, d)) {
      const int rc = ko_lines(m, &d, 1, nf, dst, 0, 1, field, koT, s);
      if (rc) return rc;
      *launches += 1;
      continue;
    }
    if (!scratch) return -4;
    char* buf = static_cast<char*>(scratch);
    const size_t nb = (size_t)m.nn * (m.precision == 0 ? sizeof(double) : sizeof(float));
    for (int q = 0; q < nf; ++q) {
      const void* src = field[q];
      for (int r = 0; r < 6; ++r) {
        void* to = buf + (r & 1) * nb;
        const int rc = launch_apply_D(m, src, to, d, s);
        if (rc) return rc;
        src = to;
      }
      const int rc = launch_axpy(m.nn, m.precision, dst[q], koT, src, s);
      if (rc) return rc;
      *launches += 7;
    }
  }
  return 0;
}

int launch_ko_fields(const DevMesh& m, int nf, void* const* out, const void* const* field, double koT, int split,
                     cudaStream_t s, int* launches) {
  const int axes[3] = {0, 1, 2};
  if (!ko_all_lines(m)) return -4;
  if (split) {
    *launches += 1;
    return ko_lines(m, axes, 3, nf, out, m.nn, 0, field, koT, s);
  }
  for (int d = 0; d < 3; ++d) {
    const int rc = ko_lines(m, axes + d, 1, nf, out, 0, d > 0, field, koT, s);
    if (rc) return rc;
  }
  *launches += 3;
  return 0;
}

}  // namespace wt
