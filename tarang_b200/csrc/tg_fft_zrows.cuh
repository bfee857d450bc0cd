// Fused z-pass for short rows, M = N3/2 in {4, 8, 16, 32}: a block takes 16 rows and runs the c2r
// transforms of all inputs side by side (one warp per input), then the r2c transforms of all
// products (one warp per product).
//
// Two lanes t = 0, 1 share a row, V = M/2 values a lane: Z[n], n = t + 2 j; DFT_V over j in
// registers, twiddle W_M^(t k1), one radix-2 butterfly between the two lanes: lane t' then holds
// z[k1 + V t'].  The forward transform is the adjoint, in the same places, so a product needs no
// exchange.  An entry and its conjugate partner M - n have the same parity, so the c2r pre-twiddle
// and the r2c post-twiddle stay inside a lane, and every twiddle but the lane's own W_2M^t is a
// compile-time constant: shared memory only carries the real-space values from the inputs' warps
// to the products' (32 consecutive entries a value, no bank conflicts).
//
// What bounds it: grids of such rows are small (32^3: 1024 rows), so the launch is a latency
// chain: two transforms deep here, NIN + NPROD in a warp that does its rows' fields in turn.
// Measured (B200, fluid, CUDA events around one launch, in brackets the radix-2 and five-stage
// shuffle kernels it replaces): 32^3 FP32 8.4 us [16.8], 64^3 FP32 10.5 [12.7], FP64 12.7 [14.7],
// 128 x 128 x 64 FP32 20.2 [27.4], FP64 29.1 [37.7].  A form with four lanes a row and V = 8, its
// exchanges through shared memory, took 15.5 us at 64^3 FP64.
#pragma once

#include "tg_fft.cuh"

namespace tg {

constexpr int kZRowsWarps = 9;  // at most one warp per product

template <typename Rw, int V>
struct ZRowLane {
  static constexpr int M = 2 * V;
  int t;
  cx<Rw> g;   // e^{+i pi t / M}
  Rw sg;      // +1 on lane 0, -1 on lane 1

  // W_M^(t k1), sign DIR: 1 on lane 0
  template <int DIR, int K>
  __device__ __forceinline__ cx<Rw> lane_tw(cx<Rw> v) const {
    const cx<Rw> w = twc<DIR, K, M, Rw>(v);
    return mkc<Rw>(t ? w.x : v.x, t ? w.y : v.y);
  }
  template <int DIR, int K>
  __device__ __forceinline__ void lane_tws(cx<Rw> (&v)[V]) const {
    if constexpr (K < V) {
      v[K] = lane_tw<DIR, K>(v[K]);
      lane_tws<DIR, K + 1>(v);
    }
  }
  // (a, b) on lanes 0, 1 -> (a + b, a - b)
  __device__ __forceinline__ void lane_bfly(cx<Rw> (&v)[V]) const {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const Rw px = __shfl_xor_sync(0xffffffffu, v[k].x, 1), py = __shfl_xor_sync(0xffffffffu, v[k].y, 1);
      v[k] = mkc<Rw>(fma(sg, v[k].x, px), fma(sg, v[k].y, py));
    }
  }
  // the slot of M - n for slot j (n = t + 2 j); slot 0 of lane 0 has its own partner `self`
  template <int J>
  __device__ __forceinline__ cx<Rw> partner(const cx<Rw> (&v)[V], cx<Rw> self) const {
    const cx<Rw> e = J == 0 ? self : v[(V - J) % V], o = v[V - 1 - J];
    return mkc<Rw>(t ? o.x : e.x, t ? o.y : e.y);
  }
  // c2r pre-twiddle (xa + conj xb) + i h (xa - conj xb), h = e^{+i pi n / M} = W_M^j g
  template <int J>
  __device__ __forceinline__ void pre(const cx<Rw> (&x)[V], cx<Rw> xM, cx<Rw> (&v)[V]) const {
    if constexpr (J < V) {
      cx<Rw> xa = x[J], xb = partner<J>(x, xM);
      if (J == 0 && t == 0) xa.y = xb.y = 0;  // the imaginary parts of X[0], X[M] are ignored
      const cx<Rw> d = mkc<Rw>(xa.x - xb.x, xa.y + xb.y);
      const cx<Rw> u = twc<+1, J, M, Rw>(g * d);
      v[J] = mkc<Rw>(xa.x + xb.x - u.y, xa.y - xb.y + u.x);
      pre<J + 1>(x, xM, v);
    }
  }
  // r2c post-twiddle hs ((z + conj zm) - i conj(h) (z - conj zm)), entries n < nout
  template <int J>
  __device__ __forceinline__ void post(const cx<Rw> (&z)[V], Rw hs, cx<Rw>* y, int nout) const {
    if constexpr (J < V) {
      const int n = t + 2 * J;
      const cx<Rw> a = z[J], b = partner<J>(z, z[0]);
      const cx<Rw> d = mkc<Rw>(a.x - b.x, a.y + b.y);
      const cx<Rw> u = twc<-1, J, M, Rw>(mkc<Rw>(fma(d.x, g.x, d.y * g.y), fma(d.y, g.x, -(d.x * g.y))));
      if (n < nout) y[n] = mkc<Rw>(hs * (a.x + b.x + u.y), hs * (a.y - b.y - u.x));
      post<J + 1>(z, hs, y, nout);
    }
  }
};

template <typename Rw, int V>
__global__ void __launch_bounds__(32 * kZRowsWarps)
    k_z_prod_rows(ZArgs a, PtrSet ps, ProdPairs pp, int nin, int nprod) {
  pdl_wait();
  constexpr int M = 2 * V;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<Rw>* rs = reinterpret_cast<cx<Rw>*>(smem_raw);  // [nin][V][32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  ZRowLane<Rw, V> L;
  L.t = lane & 1;
  L.sg = L.t ? (Rw)-1 : (Rw)1;
  L.g = conjc(cvt<Rw>(a.twN[L.t]));
  const long long row = (long long)blockIdx.x * 16 + (lane >> 1);
  const bool ok = row < a.nrows;
  for (int c = warp; c < nin; c += nw) {
    const cx<Rw>* src = reinterpret_cast<const cx<Rw>*>(ps.src[c]) + row * a.ss;
    const int nld = ok ? a.nin : 0;
    cx<Rw> x[V], v[V], xM = mkc<Rw>(0, 0);
#pragma unroll
    for (int j = 0; j < V; ++j) x[j] = (L.t + 2 * j < nld) ? src[L.t + 2 * j] : mkc<Rw>(0, 0);
    if (M < nld && L.t == 0) xM = src[M];
    L.template pre<0>(x, xM, v);
    DFT<V, +1, Rw>::run(v);
    L.template lane_tws<+1, 1>(v);
    L.lane_bfly(v);
#pragma unroll
    for (int k = 0; k < V; ++k) rs[(c * V + k) * 32 + lane] = v[k];
  }
  __syncthreads();
  const Rw sc = (Rw)a.scale, hs = (Rw)0.5 * sc;
  for (int q = warp; q < nprod; q += nw) {
    const cx<Rw>* xa = rs + pp.a[q] * V * 32 + lane;
    const cx<Rw>* xb = rs + pp.b[q] * V * 32 + lane;
    cx<Rw> v[V];
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = rmul(xa[k * 32], xb[k * 32]);
    if (pp.c[q] >= 0) {
      const cx<Rw>* xc = rs + pp.c[q] * V * 32 + lane;
      const cx<Rw>* xd = rs + pp.d[q] * V * 32 + lane;
#pragma unroll
      for (int k = 0; k < V; ++k) v[k] = v[k] - rmul(xc[k * 32], xd[k * 32]);
    }
    L.lane_bfly(v);
    L.template lane_tws<-1, 1>(v);
    DFT<V, -1, Rw>::run(v);
    if (ok) {
      cx<Rw>* dst = reinterpret_cast<cx<Rw>*>(ps.dst[q]) + row * a.ds;
      L.template post<0>(v, hs, dst, a.nout);
      if (L.t == 0 && a.nout > M) dst[M] = mkc<Rw>(sc * (v[0].x - v[0].y), (Rw)0);
      for (int k = a.nout + L.t; k < a.nfill; k += 2) dst[k] = mkc<Rw>(0, 0);
    }
  }
}

}  // namespace tg
