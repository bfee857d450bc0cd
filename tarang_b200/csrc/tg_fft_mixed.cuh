// Strided-axis c2c pass for lengths that are not powers of two: a mixed-radix Stockham FFT.
//
// A block transforms W columns of one batch of one field (a tile [L][W]).  The length is split
// into register radices (2 .. 8, 10, 12, 16) and, for what is left, prime factors of 11 and more.  Stage
// by stage, with s the product of the radices done and n = L / s what remains, n = r m:
//   y[q + s (r p + k)] = w_n^(p k) sum_j x[q + s (p + m j)] w_r^(j k),  p < m, q < s, k < r,
// which leaves the result in natural order after the last stage.  A register stage gives a thread
// one (p, q) of one column; the first reads the stored rows from global memory and the last writes
// the kept rows back, the stages between move through two shared-memory tiles.
//
// What bounds it: a pass moves each value once from and to HBM and once through shared memory per
// stage boundary, L (r1 + r2 + ..) / 2 operations a column instead of the L^2 of a direct sum.  No unit
// is near its limit (ncu, 192 x 160 x 128 FP64: HBM 14 to 30 %, FP64 pipe 13 to 16 %): at 24 % of the
// warps (127 registers) the stages' barriers, fixed latencies and loads are not hidden, and the stage
// switch has its code fetched anew by short launches.  The direct sum that this replaces was bound by
// shared-memory reads (two per multiply-add).  Measured (B200, passive scalar 96 x 80 x 64 FP64):
// y-forward of nine fields 26.9 us a launch, was 74.3; x-forward 18.8, was 58.1; y-inverse of four 17.4,
// was 55.5; a step 0.34 ms, was 0.98.
// A prime stage is a direct sum over its r inputs from shared memory, outputs k and r - k
// together: with A = x_j + x_(r-j), B = x_j - x_(r-j) they share every load and product.
#pragma once

#include "tg_fft.cuh"

namespace tg {

template <int DIR, typename R>
struct DFT<3, DIR, R> {
  __device__ __forceinline__ static void run(cx<R>* x) {
    const R s = (R)(DIR * 0.86602540378443864676);
    const cx<R> t = x[1] + x[2], d = x[1] - x[2];
    const cx<R> m = mkc<R>(x[0].x - (R)0.5 * t.x, x[0].y - (R)0.5 * t.y);
    x[0] = x[0] + t;
    x[1] = mkc<R>(m.x - s * d.y, m.y + s * d.x);
    x[2] = mkc<R>(m.x + s * d.y, m.y - s * d.x);
  }
};

// odd length N: outputs k and N - k from the sums and differences of inputs j and N - j
template <int N, int DIR, typename R>
__device__ __forceinline__ void dft_odd(cx<R>* x, const double* c, const double* s) {
  constexpr int H = (N - 1) / 2;
  cx<R> a[H], b[H];
#pragma unroll
  for (int j = 0; j < H; ++j) {
    a[j] = x[j + 1] + x[N - 1 - j];
    b[j] = x[j + 1] - x[N - 1 - j];
  }
  const cx<R> x0 = x[0];
  cx<R> t = x0;
#pragma unroll
  for (int j = 0; j < H; ++j) t = t + a[j];
  x[0] = t;
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    cx<R> u = x0, v = mkc<R>(0, 0);
#pragma unroll
    for (int j = 0; j < H; ++j) {
      const int m = ((j + 1) * k) % N;
      const R ck = (R)c[m <= H ? m : N - m];
      const R sk = (R)(DIR * (m <= H ? s[m] : -s[N - m]));
      u = mkc<R>(fma(ck, a[j].x, u.x), fma(ck, a[j].y, u.y));
      v = mkc<R>(fma(sk, b[j].x, v.x), fma(sk, b[j].y, v.y));
    }
    x[k] = mkc<R>(u.x - v.y, u.y + v.x);
    x[N - k] = mkc<R>(u.x + v.y, u.y - v.x);
  }
}
template <int DIR, typename R>
struct DFT<5, DIR, R> {
  __device__ __forceinline__ static void run(cx<R>* x) {
    constexpr double c[3] = {1.0, 0.30901699437494742410, -0.80901699437494742410};
    constexpr double s[3] = {0.0, 0.95105651629515357212, 0.58778525229247312917};
    dft_odd<5, DIR, R>(x, c, s);
  }
};
template <int DIR, typename R>
struct DFT<7, DIR, R> {
  __device__ __forceinline__ static void run(cx<R>* x) {
    constexpr double c[4] = {1.0, 0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624};
    constexpr double s[4] = {0.0, 0.78183148246802980871, 0.97492791218182360702, 0.43388373911755812048};
    dft_odd<7, DIR, R>(x, c, s);
  }
};
// coprime A, B (prime-factor map, no twiddles): n = B n1 + A n2, k = k1 mod A = k2 mod B
template <int A, int B, int DIR, typename R>
__device__ __forceinline__ void dft_pfa(cx<R>* x) {
  constexpr int N = A * B;
  cx<R> y[N];  // [k1][n2]
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
    cx<R> t[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) t[n1] = x[(B * n1 + A * n2) % N];
    DFT<A, DIR, R>::run(t);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) y[k1 * B + n2] = t[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    DFT<B, DIR, R>::run(y + k1 * B);
  }
#pragma unroll
  for (int k = 0; k < N; ++k) x[k] = y[(k % A) * B + (k % B)];
}
template <int DIR, typename R>
struct DFT<6, DIR, R> {
  __device__ __forceinline__ static void run(cx<R>* x) { dft_pfa<2, 3, DIR, R>(x); }
};
template <int DIR, typename R>
struct DFT<10, DIR, R> {
  __device__ __forceinline__ static void run(cx<R>* x) { dft_pfa<2, 5, DIR, R>(x); }
};
template <int DIR, typename R>
struct DFT<12, DIR, R> {
  __device__ __forceinline__ static void run(cx<R>* x) { dft_pfa<4, 3, DIR, R>(x); }
};

// stages of a length: register radices first (largest first, so the global loads of a thread are
// many and independent), then the primes of 11 and more
constexpr int kMixStages = 12;
struct MixPlan {
  int L = 0, ns = 0;
  int r[kMixStages] = {}, s[kMixStages] = {};  // radix; product of the radices before it
  unsigned mg[kMixStages] = {};                // ceil(2^32 / s): j / s = umulhi(j, mg) for j s < 2^32
  int wsh = 3;                                 // log2 of the columns of a tile
};
// register radix of the kernel's stage switch (the others run as prime stages)
__host__ __device__ __forceinline__ bool mix_reg_radix(int r) { return r <= 8 || r == 10 || r == 12 || r == 16; }

constexpr int kMixThreads = 128;

template <typename Ri, typename Ro, typename Rw, int DIR>
struct MixTile {
  const AxisArgs& a;
  const cx<Ri>* src;
  const cx<Ri>* src2;
  cx<Ro>* dst;
  const cx<Rw>* tw;
  int comb, col0, wsh;
  Rw sc;

  __device__ __forceinline__ cx<Rw> load(int n, int w) const {
    const int r = amap_row(a.in, n);
    cx<Rw> v = mkc<Rw>(0, 0);
    if (r >= 0 && col0 + w < a.ncols) {
      const long long o = (long long)r * a.sr + col0 + w;
      v = cvt<Rw>(src[o]);
      if (comb > 0) v = v + cvt<Rw>(src2[o]);
      else if (comb < 0) v = v - cvt<Rw>(src2[o]);
    }
    return v;
  }
  __device__ __forceinline__ void store(int k, int w, cx<Rw> v) const {
    const int r = amap_row(a.out, k);
    if (r >= 0 && col0 + w < a.ncols) dst[(long long)r * a.dr + col0 + w] = cvt<Ro>(sc * v);
  }

  template <int RR>
  __device__ __forceinline__ void reg_stage(int L, int s, unsigned mg, bool first, bool last, const cx<Rw>* x,
                                            cx<Rw>* y) const {
    const int W = 1 << wsh, m = L / (s * RR), nb = (L / RR) << wsh;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
      const int w = i & (W - 1), j = i >> wsh;
      const int p = s == 1 ? j : (int)__umulhi((unsigned)j, mg);
      const int q = j - p * s;
      cx<Rw> v[RR];
      if (first) {
#pragma unroll
        for (int k = 0; k < RR; ++k) v[k] = load(p + m * k, w);
      } else {
#pragma unroll
        for (int k = 0; k < RR; ++k) v[k] = x[((q + s * (p + m * k)) << wsh) + w];
      }
      DFT<RR, DIR, Rw>::run(v);
      if (last) {  // m = 1: no twiddles
#pragma unroll
        for (int k = 0; k < RR; ++k) store(q + s * k, w, v[k]);
      } else {
        const int e = p * s;
        y[((q + s * (RR * p)) << wsh) + w] = v[0];
#pragma unroll
        for (int k = 1; k < RR; ++k) y[((q + s * (RR * p + k)) << wsh) + w] = v[k] * tw[e * k];
      }
    }
  }

  // radix r odd prime: items (p, q) x (k = 0, or the pair k, r - k)
  __device__ __forceinline__ void prime_stage(int L, int s, unsigned mg, int r, bool last, const cx<Rw>* x,
                                              cx<Rw>* y) const {
    const int W = 1 << wsh, m = L / (s * r), H = (r + 1) / 2, nj = L / r;
    const int dtw = L / r;  // w_r = tw[L / r]
    for (int i = threadIdx.x; i < ((nj * H) << wsh); i += blockDim.x) {
      const int w = i & (W - 1), jj = i >> wsh;
      const int k = jj / nj, j = jj - k * nj;
      const int p = s == 1 ? j : (int)__umulhi((unsigned)j, mg);
      const int q = j - p * s;
      const cx<Rw>* xc = x + ((q + s * p) << wsh) + w;
      const int st = (s * m) << wsh;
      cx<Rw> u = xc[0], v = mkc<Rw>(0, 0);
      int e = 0;
      for (int t = 1; t < H; ++t) {
        const cx<Rw> g = xc[t * st], h = xc[(r - t) * st];
        e += k;
        if (e >= r) e -= r;
        const cx<Rw> c = tw[e * dtw];
        u = mkc<Rw>(fma(c.x, g.x + h.x, u.x), fma(c.x, g.y + h.y, u.y));
        v = mkc<Rw>(fma(c.y, g.x - h.x, v.x), fma(c.y, g.y - h.y, v.y));
      }
      // c.y carries the direction's sign: X_k = u + i v, X_(r-k) = u - i v
      const cx<Rw> o0 = mkc<Rw>(u.x - v.y, u.y + v.x), o1 = mkc<Rw>(u.x + v.y, u.y - v.x);
      if (last) {
        store(q + s * k, w, o0);
        if (k > 0) store(q + s * (r - k), w, o1);
      } else {
        const int e2 = p * s;
        y[((q + s * (r * p + k)) << wsh) + w] = o0 * tw[e2 * k];
        if (k > 0) y[((q + s * (r * p + r - k)) << wsh) + w] = o1 * tw[e2 * (r - k)];
      }
    }
  }
};

template <typename Ri, typename Ro, typename Rw, int DIR>
__global__ void __launch_bounds__(kMixThreads, sizeof(Rw) == 8 ? 4 : 6)
    k_axis_mixed(AxisArgs a, PtrSet ps, const __grid_constant__ MixPlan pl) {
  pdl_wait();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int L = pl.L, W = 1 << pl.wsh;
  cx<Rw>* tw = reinterpret_cast<cx<Rw>*>(smem_raw);
  cx<Rw>* x = tw + L;
  cx<Rw>* y = x + (L << pl.wsh);
  const int f = blockIdx.z;
  const int comb = a.comb[f];
  const cx<Ri>* src = reinterpret_cast<const cx<Ri>*>(ps.src[f]) + (long long)blockIdx.y * a.sb;
  const MixTile<Ri, Ro, Rw, DIR> T{
      a,
      src,
      comb ? reinterpret_cast<const cx<Ri>*>(ps.src2[f]) + (long long)blockIdx.y * a.sb : src,
      reinterpret_cast<cx<Ro>*>(ps.dst[f]) + (long long)blockIdx.y * a.db,
      tw,
      comb,
      (int)blockIdx.x * W,
      pl.wsh,
      (Rw)a.scale};
  for (int i = threadIdx.x; i < L; i += blockDim.x) {
    cx<Rw> t = cvt<Rw>(a.tw[i]);
    if (DIR > 0) t.y = -t.y;
    tw[i] = t;
  }
  if (!mix_reg_radix(pl.r[0])) {
    for (int i = threadIdx.x; i < (L << pl.wsh); i += blockDim.x) x[i] = T.load(i >> pl.wsh, i & (W - 1));
  }
  __syncthreads();
  for (int st = 0; st < pl.ns; ++st) {
    const int r = pl.r[st], s = pl.s[st];
    const unsigned mg = pl.mg[st];
    const bool first = st == 0, last = st == pl.ns - 1;
    switch (r) {
      case 2: T.template reg_stage<2>(L, s, mg, first, last, x, y); break;
      case 3: T.template reg_stage<3>(L, s, mg, first, last, x, y); break;
      case 4: T.template reg_stage<4>(L, s, mg, first, last, x, y); break;
      case 5: T.template reg_stage<5>(L, s, mg, first, last, x, y); break;
      case 6: T.template reg_stage<6>(L, s, mg, first, last, x, y); break;
      case 7: T.template reg_stage<7>(L, s, mg, first, last, x, y); break;
      case 8: T.template reg_stage<8>(L, s, mg, first, last, x, y); break;
      case 10: T.template reg_stage<10>(L, s, mg, first, last, x, y); break;
      case 12: T.template reg_stage<12>(L, s, mg, first, last, x, y); break;
      case 16: T.template reg_stage<16>(L, s, mg, first, last, x, y); break;
      default: T.prime_stage(L, s, mg, r, last, x, y); break;
    }
    __syncthreads();
    cx<Rw>* t = x;
    x = y;
    y = t;
  }
}

// The direct sum, for short lengths: a thread owns one output of a tile of eight columns.  Bound by latency: two
// trips to memory and a loop of L terms, in a kernel of few instructions, where the mixed-radix kernel fetches a
// stage's code per stage and a prime stage, with (r + 1) / 2 outputs a column, leaves most of its block idle.  The
// times of both stand at the dispatch (dft_taken).
constexpr int kDftThreads = 256;
constexpr int kDftCols = 8;
template <typename Ri, typename Ro, typename Rw, int DIR>
__global__ void __launch_bounds__(kDftThreads) k_axis_dft(AxisArgs a, PtrSet ps, int L) {
  constexpr int W = kDftCols;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<Rw>* tw = reinterpret_cast<cx<Rw>*>(smem_raw);
  cx<Rw>* tile = tw + L;  // [L][W]
  for (int i = threadIdx.x; i < L; i += kDftThreads) {
    cx<Rw> t = cvt<Rw>(a.tw[i]);
    if (DIR > 0) t.y = -t.y;
    tw[i] = t;
  }
  pdl_wait();
  const int f = blockIdx.z;
  const int comb = a.comb[f];
  const cx<Ri>* src = reinterpret_cast<const cx<Ri>*>(ps.src[f]) + (long long)blockIdx.y * a.sb;
  const cx<Ri>* src2 = comb ? reinterpret_cast<const cx<Ri>*>(ps.src2[f]) + (long long)blockIdx.y * a.sb : src;
  cx<Ro>* dst = reinterpret_cast<cx<Ro>*>(ps.dst[f]) + (long long)blockIdx.y * a.db;
  const int c0 = blockIdx.x * W;
  for (int i = threadIdx.x; i < L * W; i += kDftThreads) {
    const int r = amap_row(a.in, i / W), col = c0 + i % W;
    cx<Rw> v = mkc<Rw>(0, 0);
    if (r >= 0 && col < a.ncols) {
      const long long o = (long long)r * a.sr + col;
      v = cvt<Rw>(src[o]);
      if (comb > 0) v = v + cvt<Rw>(src2[o]);
      else if (comb < 0) v = v - cvt<Rw>(src2[o]);
    }
    tile[i] = v;
  }
  __syncthreads();
  const Rw sc = (Rw)a.scale;
  for (int i = threadIdx.x; i < L * W; i += kDftThreads) {
    const int k = i / W, w = i % W, r = amap_row(a.out, k), col = c0 + w;
    if (r < 0 || col >= a.ncols) continue;
    cx<Rw> acc = mkc<Rw>(0, 0);
    for (int n = 0, m = 0; n < L; ++n) {
      acc = acc + tile[n * W + w] * tw[m];
      m += k;
      if (m >= L) m -= L;
    }
    dst[(long long)r * a.dr + col] = cvt<Ro>(sc * acc);
  }
}

// the fewest register stages whose product is the smooth part of L, of those the ones with the
// smallest largest radix; then the primes of 11 and more.  false: more stages than a plan holds
inline bool mix_plan(int L, MixPlan& p) {
  static const int R[10] = {16, 12, 10, 8, 7, 6, 5, 4, 3, 2};
  int rest = L, best_n = kMixStages + 1, best[kMixStages] = {}, cur[kMixStages] = {};
  int primes[kMixStages], np = 0;
  int smooth = 1;
  for (int q : {2, 3, 5, 7})
    while (rest % q == 0) {
      rest /= q;
      smooth *= q;
    }
  for (int q = 11; rest > 1; q += 2)
    while (rest % q == 0) {
      if (np == kMixStages) return false;
      primes[np++] = q;
      rest /= q;
    }
  // depth-first over non-increasing radices
  struct Search {
    const int* R;
    int* best;
    int* cur;
    int& best_n;
    void go(int n, int from, int d) {
      if (n == 1) {
        if (d < best_n || (d == best_n && d > 0 && cur[0] < best[0])) {
          best_n = d;
          for (int i = 0; i < d; ++i) best[i] = cur[i];
        }
        return;
      }
      if (d >= best_n || d >= kMixStages) return;
      for (int i = from; i < 10; ++i)
        if (n % R[i] == 0) {
          cur[d] = R[i];
          go(n / R[i], i, d + 1);
        }
    }
  } search{R, best, cur, best_n};
  search.go(smooth, 0, 0);
  if (best_n > kMixStages || best_n + np > kMixStages) return false;
  p.L = L;
  p.ns = 0;
  int s = 1;
  auto add = [&](int r) {
    p.r[p.ns] = r;
    p.s[p.ns] = s;
    p.mg[p.ns] = s == 1 ? 0u : (unsigned)(((1ull << 32) + s - 1) / s);
    ++p.ns;
    s *= r;
  };
  for (int i = 0; i < best_n; ++i) add(best[i]);
  for (int i = 0; i < np; ++i) add(primes[i]);
  return true;
}

}  // namespace tg
