// Warp-level shared-memory FFTs for the resize stage of the Fourier-slice path.
//
// One warp transforms one length-n complex sequence held in shared memory,
// out of place between two buffers (Stockham autosort, natural order in and
// out).  Radices 2 to 10 and 12 have butterflies in registers; a prime factor
// above 7 takes one stage of its own (prime_stage).  Twiddles
// exp(-2 pi i m / n) are computed per launch in double precision and stored as
// float2 in shared memory.  The register FFTs (n = 32 R) copy theirs from
// tables the compiler evaluates.
//
// Sign convention: DIR = -1 is the forward transform (numpy.fft.fft),
// DIR = +1 the unnormalised inverse (n * numpy.fft.ifft).
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <new>
#include <utility>

namespace cjx {

constexpr int kMaxLength = 1026;  // the largest side and two more, a spline coefficient array's
constexpr int kMaxStages = 12;    // lengths up to that have at most 10 prime factors

struct FftPlan {
  int n;
  int nstages;  // 0 only for n = 1
  bool primes;  // a stage has a prime radix above 7 (prime_stage)
  int radix[kMaxStages];
};

// Cost of a stage of radix r over n points for one warp: the instructions of
// the rounds of 32 butterflies, each with its index arithmetic, r loads,
// twiddles and stores (about 10 per point) and the butterfly's additions and
// products, and a wait for the shared memory between two stages, which the
// one or two rounds of a short transform do not hide.  The cheapest plans of 33
// lengths from 20 to 360 were timed (cjx_fft_c2c, 2^23 points): with a wait of
// 105 to 120 instructions the plan is 0.7 % slower than the fastest on average
// and 4 % at worst, with none 3.7 % and 14 % (40 points: 5 x 2 x 4 202 us, 8 x 5
// 186 us; 54 points: 3 x 3 x 3 x 2 171 us, 9 x 6 151 us).
constexpr int kStageWait = 105;
__host__ inline int fft_stage_cost(int r, int n) {
  static const int butterfly[13] = {0, 0, 4, 14, 16, 36, 42, 70, 56, 92, 100, 0, 110};
  return kStageWait + ((n / r + 31) / 32) * (20 + 10 * r + butterfly[r]);
}

// The cheapest product of radices <= rmax that gives m; best holds the cheapest so far.
__host__ inline void fft_plan_search(int m, int rmax, int n, int cost, FftPlan& cur, FftPlan& best, int& best_cost) {
  static const int radices[] = {12, 10, 9, 8, 7, 6, 5, 4, 3, 2};
  if (cost >= best_cost) return;
  if (m == 1) {
    best = cur;
    best_cost = cost;
    return;
  }
  for (int r : radices) {
    if (r > rmax || m % r) continue;
    cur.radix[cur.nstages++] = r;
    fft_plan_search(m / r, r, n, cost + fft_stage_cost(r, n), cur, best, best_cost);
    --cur.nstages;
  }
}

// Bound by instructions.  512 images 180^2 from N = 360 (5 x 6 x 12 and
// 5 x 6 x 6 instead of 8 x 5 x 3 x 3 and 4 x 5 x 3 x 3; a multiplication in
// place of the two divisions per butterfly; a quadrant of twiddles evaluated
// instead of all; image constants once per CTA; held to 64 registers for 4
// CTAs per SM): the three resize passes 321 + 252 + 194 us before, 206 + 157 +
// 149 us with all of that.
// Prime factors above 7 first, then the odd radices, then the even ones in
// ascending order: a stage stores at stride (product of the earlier radices)
// x its own radix, so an odd first radix keeps the first stores free of bank
// conflicts and a later even one starts from runs of consecutive entries.
// A plan of two stages starts with its larger radix, whose twiddles are all 1
// there (50 points: 10 x 5 165 us, 5 x 10 181 us).
__host__ inline FftPlan search_fft_plan(int n) {
  FftPlan p{};
  p.n = n;
  int m = n;
  for (int f : {2, 3, 5, 7})
    while (m % f == 0) m /= f;
  const int smooth = n / m;
  for (int f = 11; m > 1; f += 2)
    while (m % f == 0) {
      p.radix[p.nstages++] = f;
      p.primes = true;
      m /= f;
    }
  FftPlan cur{}, best{};
  int best_cost = 1 << 30;
  fft_plan_search(smooth, 12, n, 0, cur, best, best_cost);
  if (best.nstages == 2 && p.nstages == 0) {
    for (int s = 0; s < 2; ++s) p.radix[p.nstages++] = best.radix[s];
    return p;
  }
  for (int odd = 1; odd >= 0; --odd)
    for (int s = best.nstages - 1; s >= 0; --s)
      if ((best.radix[s] & 1) == odd) p.radix[p.nstages++] = best.radix[s];
  return p;
}

// The plan of a length, searched once per process (60 bytes each, at most one
// per length): every call of the library makes three.  cjx_slice_ctf_workspace_size
// from Python: 2.5 us with the fixed order of radices, 3.2 to 5.7 with a search
// per call, 2.6 with the table.
__host__ inline FftPlan make_fft_plan(int n) {
  static std::atomic<const FftPlan*> known[kMaxLength + 1];
  if (n < 1 || n > kMaxLength) return search_fft_plan(n);
  const FftPlan* plan = known[n].load(std::memory_order_acquire);
  if (plan) return *plan;
  const FftPlan made = search_fft_plan(n);
  const FftPlan* mine = new (std::nothrow) FftPlan(made);
  if (mine && !known[n].compare_exchange_strong(plan, mine, std::memory_order_acq_rel)) delete mine;  // another thread's
  return made;
}

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
// multiply by DIR * i
template <int DIR>
__device__ __forceinline__ float2 cmul_i(float2 a) {
  return DIR > 0 ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}
// twiddle exp(DIR * 2 pi i m / n) from the forward table
template <int DIR>
__device__ __forceinline__ float2 twiddle(const float2* tw, int m) {
  float2 w = tw[m];
  return DIR > 0 ? cconj(w) : w;
}

// Fill tw[m] = exp(-2 pi i m / n), m in [0, n), cooperatively by the block.
// One quadrant (or half) is evaluated and turned into the others, which gives
// the same bits: sincospi reduces its argument by quadrants exactly.
__device__ inline void build_twiddles(float2* tw, int n) {
  const int parts = (n % 4 == 0) ? 4 : (n % 2 == 0) ? 2 : 1, len = n / parts;
  for (int m = threadIdx.x; m < len; m += blockDim.x) {
    double s, c;
    sincospi(-2.0 * (double)m / (double)n, &s, &c);
    const float2 w = make_float2((float)c, (float)s);
    tw[m] = w;
    if (parts > 1) tw[m + n / 2] = make_float2(-w.x, -w.y);
    if (parts == 4) {  // times -i, times +i
      tw[m + len] = make_float2(w.y, -w.x);
      tw[m + 3 * len] = make_float2(-w.y, w.x);
    }
  }
}

template <int DIR>
__device__ __forceinline__ void dft2(float2* v) {
  float2 a = v[0];
  v[0] = cadd(a, v[1]);
  v[1] = csub(a, v[1]);
}

template <int DIR>
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3) {
  float2 s02 = cadd(a0, a2), d02 = csub(a0, a2);
  float2 s13 = cadd(a1, a3), d13 = csub(a1, a3);
  float2 t = cmul_i<DIR>(d13);
  a0 = cadd(s02, s13);
  a2 = csub(s02, s13);
  a1 = cadd(d02, t);
  a3 = csub(d02, t);
}

template <int DIR>
__device__ __forceinline__ void dft3(float2* v) {
  const float c = 0.86602540378443864676f;  // sqrt(3)/2
  float2 s = cadd(v[1], v[2]), d = csub(v[1], v[2]);
  float2 x0 = cadd(v[0], s);
  float2 m = make_float2(fmaf(-0.5f, s.x, v[0].x), fmaf(-0.5f, s.y, v[0].y));
  float2 t = cscale(cmul_i<DIR>(d), c);
  v[0] = x0;
  v[1] = cadd(m, t);
  v[2] = csub(m, t);
}

template <int DIR>
__device__ __forceinline__ void dft5(float2* v) {
  const float c1 = 0.30901699437494742410f;   // cos(2 pi / 5)
  const float c2 = -0.80901699437494742410f;  // cos(4 pi / 5)
  const float s1 = 0.95105651629515357212f;   // sin(2 pi / 5)
  const float s2 = 0.58778525229247312917f;   // sin(4 pi / 5)
  float2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
  float2 t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
  float2 a0 = v[0];
  float2 m1 = make_float2(a0.x + c1 * t1.x + c2 * t2.x, a0.y + c1 * t1.y + c2 * t2.y);
  float2 m2 = make_float2(a0.x + c2 * t1.x + c1 * t2.x, a0.y + c2 * t1.y + c1 * t2.y);
  float2 n1 = cmul_i<DIR>(make_float2(s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y));
  float2 n2 = cmul_i<DIR>(make_float2(s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y));
  v[0] = cadd(a0, cadd(t1, t2));
  v[1] = cadd(m1, n1);
  v[4] = csub(m1, n1);
  v[2] = cadd(m2, n2);
  v[3] = csub(m2, n2);
}

template <int DIR>
__device__ __forceinline__ void dft8(float2* v) {
  const float r = 0.70710678118654752440f;
  float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
  float2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  dft4<DIR>(e0, e1, e2, e3);
  dft4<DIR>(o0, o1, o2, o3);
  // o_k *= exp(DIR 2 pi i k / 8)
  o1 = make_float2((o1.x - DIR * o1.y) * r, (o1.y + DIR * o1.x) * r);
  o2 = cmul_i<DIR>(o2);
  o3 = make_float2((-o3.x - DIR * o3.y) * r, (-o3.y + DIR * o3.x) * r);
  v[0] = cadd(e0, o0);
  v[4] = csub(e0, o0);
  v[1] = cadd(e1, o1);
  v[5] = csub(e1, o1);
  v[2] = cadd(e2, o2);
  v[6] = csub(e2, o2);
  v[3] = cadd(e3, o3);
  v[7] = csub(e3, o3);
}

// ===========================================================================
// Register FFT for n = 32 R (R in {1, 2, 3, 4, 5, 6, 8, 10, 12, 16}).
//
// Four-step split n = 32 n1 + n2, k = k1 + R k2 (n2, k2 across the 32 lanes;
// n1, k1 in registers):
//   X[k1 + R k2] = sum_n2 W_32^(n2 k2) W_n^(n2 k1) sum_n1 x[32 n1 + n2] W_R^(n1 k1)
// 1. lane l holds x[32 n1 + brev5(l)] for n1 = 0..R-1 (the caller loads them);
// 2. R-point DFT over n1 in registers (compile-time twiddles);
// 3. multiply by W_n^(brev5(l) k1) from a [R][32] table (conflict-free);
// 4. 32-point radix-2 decimation-in-time across lanes with warp shuffles;
//    bit-reversed lane order in, natural order out.
// Afterwards lane l holds X[k1 + R l] for k1 = 0..R-1.
// Shared-memory buffers that receive these outputs use the padded layout
// pad16(e) = e + e / 16, which keeps the stride-R stores near conflict-free.
// ===========================================================================

__host__ __device__ constexpr int pad16(int e) { return e + (e >> 4); }

__device__ __forceinline__ int brev5(int l) { return (int)(__brev((unsigned)l) >> 27); }

// Shared-memory staging of a register FFT's outputs (lane l holds k = k1 + R l)
// for reading back in natural order.  pad16 is conflict-free for the
// power-of-two R; for R = 10 (the 320-point transforms) its stride-10 stores
// meet 5-way bank conflicts within a half-warp, and k + k/16 + 14 (k/32) keeps
// both the stores and the natural-order reads conflict-free (20 + 32
// wavefronts per 320 outputs against 100 + 32, counted on the CPU).
__host__ __device__ constexpr int stage_r(int R, int k) { return R == 10 ? k + (k >> 4) + (k >> 5) * 14 : pad16(k); }
__host__ __device__ constexpr int stage_r_size(int R) { return stage_r(R, 32 * R - 1) + 1; }
// The same for warp_fft512_t's outputs (k = fft512_t_out(q, lane)): its two
// lane halves land 256 apart and, with pad16 alone, on the same banks; the
// second half moves by 8 entries.  Size 551.
__host__ __device__ constexpr int stage512(int k) { return pad16(k) + 8 * ((k >> 8) & 1); }
constexpr int kStage512Size = 551;

// Compile-time cos / sin of 2 pi m / R via Taylor series after reduction to
// |x| <= pi/4 (enough terms for double precision); used only for the small
// constant twiddles of the in-register DFTs.
namespace ct {
constexpr double kPi = 3.14159265358979323846264338327950288;
constexpr double taylor_sin(double x) {
  double term = x, sum = x;
  for (int k = 1; k < 14; ++k) {
    term *= -x * x / ((2.0 * k) * (2.0 * k + 1.0));
    sum += term;
  }
  return sum;
}
constexpr double taylor_cos(double x) {
  double term = 1.0, sum = 1.0;
  for (int k = 1; k < 14; ++k) {
    term *= -x * x / ((2.0 * k - 1.0) * (2.0 * k));
    sum += term;
  }
  return sum;
}
// angle = 2 pi m / R reduced by octant symmetry
constexpr double cos2pi(int m, int R) {
  m = ((m % R) + R) % R;
  const double x = 2.0 * kPi * m / R;  // [0, 2 pi)
  if (x <= kPi / 4) return taylor_cos(x);
  if (x <= 3 * kPi / 4) return -taylor_sin(x - kPi / 2);
  if (x <= 5 * kPi / 4) return -taylor_cos(x - kPi);
  if (x <= 7 * kPi / 4) return taylor_sin(x - 3 * kPi / 2);
  return taylor_cos(x - 2 * kPi);
}
constexpr double sin2pi(int m, int R) { return cos2pi(m * 4 - R, 4 * R); }

// Register-FFT twiddle tables, evaluated by the compiler: for each n = 32 R
// with R in the register-FFT list, entries k1 * 32 + l = exp(-2 pi i brev5(l)
// k1 / n) (the layout build_reg_twiddles fills), back to back in the order
// of that list; then w32[m] = exp(-2 pi i m / 32).
__host__ __device__ constexpr int reg_table_offset(int R) {
  switch (R) {
    case 1: return 0;
    case 2: return 32;
    case 3: return 96;
    case 4: return 192;
    case 5: return 320;
    case 6: return 480;
    case 8: return 672;
    case 10: return 928;
    case 12: return 1248;
    case 16: return 1632;
    default: return -1;
  }
}
constexpr int kRegTableSize = 2144;  // 32 * (1 + 2 + 3 + 4 + 5 + 6 + 8 + 10 + 12 + 16)
constexpr int brev5c(int l) {
  int r = 0;
  for (int b = 0; b < 5; ++b) r |= ((l >> b) & 1) << (4 - b);
  return r;
}
struct TwiddleTables {
  float2 reg[kRegTableSize];
  float2 w32[32];
};
constexpr TwiddleTables make_twiddle_tables() {
  TwiddleTables t{};
  const int radices[10] = {1, 2, 3, 4, 5, 6, 8, 10, 12, 16};
  for (int q = 0; q < 10; ++q) {
    const int R = radices[q], n = 32 * R, o = reg_table_offset(R);
    for (int k1 = 0; k1 < R; ++k1)
      for (int l = 0; l < 32; ++l) {
        const int a = brev5c(l) * k1;
        t.reg[o + k1 * 32 + l] = float2{(float)cos2pi(a, n), (float)-sin2pi(a, n)};
      }
  }
  for (int m = 0; m < 32; ++m) t.w32[m] = float2{(float)cos2pi(m, 32), (float)-sin2pi(m, 32)};
  return t;
}
}  // namespace ct

// In global memory (L2-resident after the first CTAs): every CTA copies its
// table into shared memory instead of evaluating n double-precision sincospi.
// Not declared const, so that it stays an ordinary global array read through
// the L1 (lanes read different entries).
static __device__ ct::TwiddleTables kTwiddleTables = ct::make_twiddle_tables();

// exp(DIR 2 pi i m / R) as a compile-time constant
template <int DIR, int M, int R>
__device__ __forceinline__ float2 ctw() {
  constexpr float c = (float)ct::cos2pi(M, R);
  constexpr float s = (float)ct::sin2pi(M, R);
  return make_float2(c, DIR > 0 ? s : -s);
}

template <int DIR, int M, int R>
__device__ __forceinline__ float2 ctw_mul(float2 v) {
  if constexpr ((M % R) == 0) {
    return v;
  } else {
    return cmul(v, ctw<DIR, M, R>());
  }
}

template <int R, int DIR>
struct RegDft;

template <int DIR>
struct RegDft<1, DIR> {
  __device__ __forceinline__ static void run(float2*) {}
};
template <int DIR>
struct RegDft<2, DIR> {
  __device__ __forceinline__ static void run(float2* v) { dft2<DIR>(v); }
};
template <int DIR>
struct RegDft<3, DIR> {
  __device__ __forceinline__ static void run(float2* v) { dft3<DIR>(v); }
};
template <int DIR>
struct RegDft<4, DIR> {
  __device__ __forceinline__ static void run(float2* v) { dft4<DIR>(v[0], v[1], v[2], v[3]); }
};
template <int DIR>
struct RegDft<5, DIR> {
  __device__ __forceinline__ static void run(float2* v) { dft5<DIR>(v); }
};
template <int DIR>
struct RegDft<7, DIR> {  // pairs (r, 7 - r): real factors, X[q] and X[7 - q] from the same products
  __device__ __forceinline__ static void run(float2* v) {
    constexpr float c[4] = {1.0f, (float)ct::cos2pi(1, 7), (float)ct::cos2pi(2, 7), (float)ct::cos2pi(3, 7)};
    constexpr float d[4] = {0.0f, (float)ct::sin2pi(1, 7), (float)ct::sin2pi(2, 7), (float)ct::sin2pi(3, 7)};
    const float2 x0 = v[0];
    const float2 s1 = cadd(v[1], v[6]), s2 = cadd(v[2], v[5]), s3 = cadd(v[3], v[4]);
    const float2 d1 = csub(v[1], v[6]), d2 = csub(v[2], v[5]), d3 = csub(v[3], v[4]);
    v[0] = cadd(cadd(x0, s1), cadd(s2, s3));
    pair(v[1], v[6], x0, s1, s2, s3, c[1], c[2], c[3], d1, d2, d3, d[1], d[2], d[3]);
    pair(v[2], v[5], x0, s1, s2, s3, c[2], c[3], c[1], d1, d2, d3, d[2], -d[3], -d[1]);
    pair(v[3], v[4], x0, s1, s2, s3, c[3], c[1], c[2], d1, d2, d3, d[3], -d[1], d[2]);
  }
  __device__ __forceinline__ static void pair(float2& up, float2& down, float2 x0, float2 s1, float2 s2, float2 s3,
                                              float c1, float c2, float c3, float2 d1, float2 d2, float2 d3, float e1,
                                              float e2, float e3) {
    const float2 a = make_float2(fmaf(c3, s3.x, fmaf(c2, s2.x, fmaf(c1, s1.x, x0.x))),
                                 fmaf(c3, s3.y, fmaf(c2, s2.y, fmaf(c1, s1.y, x0.y))));
    const float2 b = cmul_i<DIR>(make_float2(fmaf(e3, d3.x, fmaf(e2, d2.x, e1 * d1.x)),
                                             fmaf(e3, d3.y, fmaf(e2, d2.y, e1 * d1.y))));
    up = cadd(a, b);
    down = csub(a, b);
  }
};
template <int DIR>
struct RegDft<8, DIR> {
  __device__ __forceinline__ static void run(float2* v) { dft8<DIR>(v); }
};

// R = A * B: X[kA + A kB] = sum_b W_B^(b kB) W_R^(b kA) sum_a v[B a + b] W_A^(a kA)
template <int A, int B, int DIR>
struct RegDftAB {
  template <int b, int kA>
  __device__ __forceinline__ static void twiddle_one(float2 (&u)[B][A]) {
    u[b][kA] = ctw_mul<DIR, b * kA, A * B>(u[b][kA]);
  }
  template <int b, int... kA>
  __device__ __forceinline__ static void twiddle_row(float2 (&u)[B][A], std::integer_sequence<int, kA...>) {
    (twiddle_one<b, kA>(u), ...);
  }
  template <int... b>
  __device__ __forceinline__ static void twiddle_all(float2 (&u)[B][A], std::integer_sequence<int, b...>) {
    (twiddle_row<b>(u, std::make_integer_sequence<int, A>{}), ...);
  }
  __device__ __forceinline__ static void run(float2* v) {
    float2 u[B][A];
#pragma unroll
    for (int b = 0; b < B; ++b) {
#pragma unroll
      for (int a = 0; a < A; ++a) u[b][a] = v[B * a + b];
      RegDft<A, DIR>::run(u[b]);
    }
    twiddle_all(u, std::make_integer_sequence<int, B>{});
#pragma unroll
    for (int kA = 0; kA < A; ++kA) {
      float2 w[B];
#pragma unroll
      for (int b = 0; b < B; ++b) w[b] = u[b][kA];
      RegDft<B, DIR>::run(w);
#pragma unroll
      for (int kB = 0; kB < B; ++kB) v[kA + A * kB] = w[kB];
    }
  }
};

template <int DIR>
struct RegDft<6, DIR> : RegDftAB<2, 3, DIR> {};
template <int DIR>
struct RegDft<10, DIR> : RegDftAB<2, 5, DIR> {};
template <int DIR>
struct RegDft<9, DIR> : RegDftAB<3, 3, DIR> {};
template <int DIR>
struct RegDft<12, DIR> : RegDftAB<4, 3, DIR> {};
template <int DIR>
struct RegDft<16, DIR> : RegDftAB<4, 4, DIR> {};

// ===========================================================================
// Shared-memory FFT of any length up to CJX_MAX_SIDE.
// ===========================================================================

// j / d for j < 1024 and d in [1, 1024] by one multiplication with
// div_inverse(d): ceil(2^21 / d) d - 2^21 < d, and j d <= 2^20.
__device__ __forceinline__ unsigned div_inverse(int d) { return ((1u << 21) + (unsigned)d - 1u) / (unsigned)d; }
__device__ __forceinline__ int div_by(int j, unsigned inverse) { return (int)(((unsigned)j * inverse) >> 21); }

template <int R, int DIR>
__device__ __forceinline__ void stockham_stage(const float2* __restrict__ in, float2* __restrict__ out,
                                               int n, int Ns, const float2* tw, int lane) {
  const int nb = n / R;
  const int tstep = n / (Ns * R);
  const unsigned inv = div_inverse(Ns);
  for (int j = lane; j < nb; j += 32) {
    const int g = div_by(j, inv), k = j - g * Ns;
    float2 v[R];
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = in[j + q * nb];
    if (Ns > 1) {  // q k tstep < n
      const float2* w = tw;
#pragma unroll
      for (int q = 1; q < R; ++q) {
        w += k * tstep;
        v[q] = cmul(v[q], twiddle<DIR>(w, 0));
      }
    }
    RegDft<R, DIR>::run(v);
    float2* o = out + g * Ns * R + k;
#pragma unroll
    for (int q = 0; q < R; ++q) o[q * Ns] = v[q];
  }
}

// Stage of a prime radix p > 7, in two steps.  First every pair of inputs
// (r, p - r) is replaced by its sum and difference (in overwrites itself);
// then X[q] and X[p - q] come from the same products,
//   X[q], X[p - q] = x_0 + sum_r s_r cos(2 pi r q / p) +- i sum_r d_r sin(...),
// real factors on (p - 1) / 2 pairs: a quarter of the multiplications of the
// direct sum.  A lane keeps Q outputs, so that each pair read serves all of them.
// Unrolled by 4: 1021 points 1.51 ms, 1.67 ms without.
template <int Q, int DIR>
__device__ __forceinline__ void prime_outputs(const float2* __restrict__ in, float2* __restrict__ out, int n, int p,
                                              int Ns, const float2* tw, int lane) {
  const int nb = n / p, half = (p - 1) / 2, groups = half / Q + 1;
  const unsigned inv_nb = div_inverse(nb), inv_ns = div_inverse(Ns);
  for (int t = lane; t < nb * groups; t += 32) {
    const int qg = div_by(t, inv_nb), j = t - qg * nb;
    const float2 x0 = in[j];
    float2 A[Q], B[Q];
    int m[Q], step[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      A[i] = x0;
      B[i] = make_float2(0.f, 0.f);
      m[i] = 0;
      step[i] = min(Q * qg + i, half) * nb;
    }
    const float2* lo = in + j;
    const float2* hi = in + j + n;
#pragma unroll 4
    for (int r = 1; r <= half; ++r) {
      lo += nb;
      hi -= nb;
      const float2 s = *lo, d = *hi;
#pragma unroll
      for (int i = 0; i < Q; ++i) {
        m[i] += step[i];
        if (m[i] >= n) m[i] -= n;
        const float2 w = tw[m[i]];
        A[i].x = fmaf(s.x, w.x, A[i].x);
        A[i].y = fmaf(s.y, w.x, A[i].y);
        B[i].x = fmaf(d.x, w.y, B[i].x);
        B[i].y = fmaf(d.y, w.y, B[i].y);
      }
    }
    const int g = div_by(j, inv_ns);
    float2* o = out + g * Ns * p + (j - g * Ns);
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const int q = Q * qg + i;
      const float2 b = DIR < 0 ? make_float2(-B[i].y, B[i].x) : make_float2(B[i].y, -B[i].x);
      if (q <= half) o[q * Ns] = cadd(A[i], b);
      if (q > 0 && q <= half) o[(p - q) * Ns] = csub(A[i], b);
    }
  }
}

template <int DIR>
__device__ __forceinline__ void prime_stage(float2* __restrict__ in, float2* __restrict__ out, int n, int p, int Ns,
                                            const float2* tw, int lane) {
  const int nb = n / p, half = (p - 1) / 2;
  const int tstep = n / (Ns * p);
  const unsigned inv_nb = div_inverse(nb), inv_ns = div_inverse(Ns);
  for (int e = lane; e < nb * half; e += 32) {
    const int r = 1 + div_by(e, inv_nb), j = e - (r - 1) * nb;
    const int k = j - div_by(j, inv_ns) * Ns;
    float2 a = in[j + r * nb], b = in[j + (p - r) * nb];
    if (Ns > 1) {
      a = cmul(a, twiddle<DIR>(tw, r * k * tstep));
      b = cmul(b, twiddle<DIR>(tw, (p - r) * k * tstep));
    }
    in[j + r * nb] = cadd(a, b);
    in[j + (p - r) * nb] = csub(a, b);
  }
  __syncwarp();
  // Rounds of 32 lanes: four outputs each take three times as long as one.  2^23 points with one, with four: 101
  // points 237 us, 309 (2 rounds, 1); 163 points 314, 309 (3, 1); 202 points 207, 184 (4, 1); 262 points 240, 287 (5,
  // 2); 340 points 98, 92 (6, 2); 676 points 117, 110 (12, 4).  Of 60 lengths the slower one is chosen at four, by
  // at most 6 %.
  if (3 * ((nb * (half / 4 + 1) + 31) / 32) <= (nb * (half + 1) + 31) / 32)
    prime_outputs<4, DIR>(in, out, n, p, Ns, tw, lane);
  else
    prime_outputs<1, DIR>(in, out, n, p, Ns, tw, lane);
}

// Transform buffer `a` (length plan.n) with scratch `b`; returns the buffer
// holding the result (a or b).  Executed by one full warp; ends with __syncwarp.
// PRIMES: the plan may have prime stages (plan.primes).  Every kernel has an
// instance without them for the other lengths, held to 64 registers (4 CTAs
// per SM), one with them that may take more, and a __grid_constant__ plan, which is
// indexed in place instead of copied to local memory.  With prime_stage as a
// call in a single instance, 80 registers: 48 points 195 us (cjx_fft_c2c, 2^23
// points) before prime stages existed, 208 with the
// call, 160 now (plan included); 360 points 90, 71, 62; 101 points 630, 243, 240; 1021 points
// 5760, 1414, 1513.  Ewald rows of 1024 images 48^2 from N = 96: 99, 109, 91.
template <int DIR, bool PRIMES>
__device__ __forceinline__ float2* warp_fft(float2* a, float2* b, const FftPlan& plan, const float2* tw, int lane) {
  const int n = plan.n;
  if (plan.nstages == 0) {  // n = 1
    if (lane == 0) b[0] = a[0];
    __syncwarp();
    return b;
  }
  int Ns = 1;
  for (int s = 0; s < plan.nstages; ++s) {
    const int R = plan.radix[s];
    switch (R) {
      case 2: stockham_stage<2, DIR>(a, b, n, Ns, tw, lane); break;
      case 3: stockham_stage<3, DIR>(a, b, n, Ns, tw, lane); break;
      case 4: stockham_stage<4, DIR>(a, b, n, Ns, tw, lane); break;
      case 5: stockham_stage<5, DIR>(a, b, n, Ns, tw, lane); break;
      case 6: stockham_stage<6, DIR>(a, b, n, Ns, tw, lane); break;
      case 7: stockham_stage<7, DIR>(a, b, n, Ns, tw, lane); break;
      case 8: stockham_stage<8, DIR>(a, b, n, Ns, tw, lane); break;
      case 9: stockham_stage<9, DIR>(a, b, n, Ns, tw, lane); break;
      case 10: stockham_stage<10, DIR>(a, b, n, Ns, tw, lane); break;
      case 12: stockham_stage<12, DIR>(a, b, n, Ns, tw, lane); break;
      default:
        if constexpr (PRIMES) prime_stage<DIR>(a, b, n, R, Ns, tw, lane);
        break;
    }
    __syncwarp();
    float2* t = a;
    a = b;
    b = t;
    Ns *= R;
  }
  return a;
}

// Per-lane twiddles of the 5 cross-lane DIT stages (forward sign):
// stage s (span h = 2^s) uses exp(-2 pi i (l mod h) / (2h)) =
// W32[(l mod h) * 16 / h].  Only upper lanes (bit h set) use them.
struct LaneTwiddles {
  float2 w[5];
};

// w32[m] = exp(-2 pi i m / 32), m in [0, 32) (block-cooperative).
__device__ inline void build_w32(float2* w32) {
  if (threadIdx.x < 32) w32[threadIdx.x] = __ldg(&kTwiddleTables.w32[threadIdx.x]);
}

__device__ __forceinline__ LaneTwiddles make_lane_twiddles(const float2* w32, int lane) {
  LaneTwiddles t;
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int h = 1 << s;
    t.w[s] = (lane & h) ? w32[(lane & (h - 1)) * (16 >> s)] : make_float2(1.f, 0.f);
  }
  return t;
}

// Fill tab[k1 * 32 + l] = exp(-2 pi i brev5(l) k1 / n), k1 in [0, R) (block-cooperative).
__device__ inline void build_reg_twiddles(float2* tab, int n) {
  const int R = n / 32;
  const int o = (n % 32 == 0) ? ct::reg_table_offset(R) : -1;
  if (o >= 0) {
    for (int e = threadIdx.x; e < n; e += blockDim.x) tab[e] = __ldg(&kTwiddleTables.reg[o + e]);
    return;
  }
  for (int e = threadIdx.x; e < R * 32; e += blockDim.x) {
    const int k1 = e >> 5, l = e & 31;
    double s, c;
    sincospi(-2.0 * (double)(brev5(l) * k1) / (double)n, &s, &c);
    tab[e] = make_float2((float)c, (float)s);
  }
}

// Steps 2-4 on the lane's R values (step 1 input already loaded).
// Cross-lane DIT butterfly: the upper lane pre-multiplies its value by the
// stage twiddle (lower lanes hold w = 1), the pair exchanges values, then
// lower = own + partner and upper = partner - own.
template <int R, int DIR>
__device__ __forceinline__ void warp_fft_reg(float2 (&x)[R], const float2* __restrict__ tab, const LaneTwiddles& lt,
                                             int lane) {
  RegDft<R, DIR>::run(x);
#pragma unroll
  for (int k1 = 1; k1 < R; ++k1) x[k1] = cmul(x[k1], twiddle<DIR>(tab, k1 * 32 + lane));
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const int h = 1 << s;
    const float sg = (lane & h) ? -1.f : 1.f;
    const float2 w = DIR > 0 ? cconj(lt.w[s]) : lt.w[s];
#pragma unroll
    for (int k1 = 0; k1 < R; ++k1) {
      float2 v = (s == 0) ? x[k1] : cmul(x[k1], w);
      float2 p;
      p.x = __shfl_xor_sync(0xffffffffu, v.x, h);
      p.y = __shfl_xor_sync(0xffffffffu, v.y, h);
      x[k1] = make_float2(fmaf(sg, v.x, p.x), fmaf(sg, v.y, p.y));
    }
  }
}

// Sizes the register FFT handles: n = 32 R with R in the list above.
__host__ __device__ inline int reg_fft_radix(int n) {
  if (n % 32 != 0) return 0;
  const int R = n / 32;
  switch (R) {
    case 1: case 2: case 3: case 4: case 5: case 6: case 8: case 10: case 12: case 16:
      return R;
    default:
      return 0;
  }
}

// 512-point warp FFT as 16 x 32 with one shared-memory transpose:
// x[n] = x[l + 32 n1] (l = lane), X[k] = X[k1 + 16 k2].
//   1. a 16-point DFT over n1 in registers, twiddle W_512^(l k1);
//   2. transpose through shared memory so that lane (k1, e) = (lane >> 1,
//      lane & 1) holds the 16 values z[2m + e] of column k1;
//   3. a 16-point DFT over m in registers (the even / odd half of the
//      32-point DFT over l), then one cross-lane radix-2 step with W_32^q:
//      X[k1 + 16 q] = Y0 + W Y1 (e = 0), X[k1 + 16 (q + 16)] = Y0 - W Y1 (e = 1).
// About 40 % fewer instructions than the five-shuffle-stage network of
// warp_fft_reg<16> (32 shuffles per lane instead of 160).
// Input: x[n1] = data[32 n1 + lane] (natural lane order, unlike
// warp_fft_reg).  Output: x[q] = X[fft512_t_out(q, lane)].  tab is the
// build_reg_twiddles(n = 512) table, w32 the build_w32 table, scr a
// per-warp shared buffer of >= 16 * 34 values (overwritten).
__device__ __forceinline__ int fft512_t_out(int q, int lane) { return (lane >> 1) + 16 * (q + 16 * (lane & 1)); }

template <int DIR>
__device__ __forceinline__ void warp_fft512_t(float2 (&x)[16], const float2* __restrict__ tab,
                                              const float2* __restrict__ w32, float2* __restrict__ scr, int lane) {
  constexpr int kStride = 34;  // row stride: conflict-free 8-byte reads within each half-warp
  RegDft<16, DIR>::run(x);
  const int bl = brev5(lane);
#pragma unroll
  for (int k1 = 1; k1 < 16; ++k1) x[k1] = cmul(x[k1], twiddle<DIR>(tab, k1 * 32 + bl));  // W_512^(lane k1)
#pragma unroll
  for (int k1 = 0; k1 < 16; ++k1) scr[k1 * kStride + lane] = x[k1];
  __syncwarp();
  const int c = lane >> 1, e = lane & 1;
#pragma unroll
  for (int m = 0; m < 16; ++m) x[m] = scr[c * kStride + 2 * m + e];
  __syncwarp();
  RegDft<16, DIR>::run(x);
  const float sg = e ? -1.f : 1.f;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    float2 w = e ? w32[q] : make_float2(1.f, 0.f);
    if (DIR > 0) w = cconj(w);
    const float2 v = cmul(x[q], w);
    float2 p;
    p.x = __shfl_xor_sync(0xffffffffu, v.x, 1);
    p.y = __shfl_xor_sync(0xffffffffu, v.y, 1);
    x[q] = make_float2(fmaf(sg, v.x, p.x), fmaf(sg, v.y, p.y));
  }
}

}  // namespace cjx
