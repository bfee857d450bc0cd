// y-inverse, z-pass (c2r, products, r2c) and y-forward of one x-plane in shared memory, for planes that fit
// there: N2 and N3 of 32 or 64.
//
// After the x-inverse the planes are independent up to the x-forward, so a block carries one plane of all
// fields through: y columns of the inputs from global memory (radix R1, then R2, in place), two lanes a z
// row (ZRowLane, in place), the products' rows into buffers of their own, their y columns, the last radix
// straight to global memory.  The y order between the two halves of a transform is the digit-reversed one:
// the z-pass and the products act row by row, and the forward transform is the adjoint, so nothing is
// reordered.  Row strides are 2 modulo 4 elements: the two lanes of neighbouring rows fall into different
// banks, and lanes along a row do anyway.
//
// What bounds it: a lone grid of this size has 32 or 64 planes, so the kernel is a latency chain of six phases,
// at 64 x 64 the instructions of one SM's share; it saves two launches a stage and the intermediates' four trips
// through L2, for a batch through HBM.
// Measured (B200, FP32-mixed step, against the y, z and y passes one by one): 32^3 fluid 51.4 us [59.8], 64^3 76.2
// [80.8]; a step of one of 64 batched requests 32^3 fluid 4.9 us [6.6], 64^3 25.9 [30.0], 64^3 MHD 54.6 [56.7].
// Four blocks a plane gained nothing over two (the first radix is computed by each of them).
#include "tg_plane.h"

#include <algorithm>

#include <cooperative_groups.h>

#include "tg_fft_zrows.cuh"

namespace cg = cooperative_groups;

namespace tg {

namespace {

constexpr size_t kPlaneSmem = 227 * 1024;

template <typename R>
struct PlaneThreads {
  static constexpr int v = sizeof(R) == 8 ? 320 : 640;  // the most a block has (register bound)
};

// C: blocks (a cluster) that share a plane.  Block c takes the y rows with k1 / (R1 / C) = c: the first radix
// of the y-inverse is computed by each for its own k1, all is local from there, and only the last radix of
// the y-forward reads the other blocks' slots.
template <typename R, int R1, int R2, int V, int C>
__global__ void __launch_bounds__(PlaneThreads<R>::v) k_plane(PlaneArgs a, PtrSet ps, ProdPairs pp) {
  constexpr int N2 = R1 * R2, M = 2 * V, KC = R1 / C, NR = N2 / C;  // NR: rows of the block
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cx<R>* tw = reinterpret_cast<cx<R>*>(smem_raw);  // [N2]
  cx<R>* in = tw + N2;                             // [nin][NR][rin]
  cx<R>* out = in + a.nin * NR * a.rin;            // [nprod][NR][rout]
  const int tid = threadIdx.x, T = blockDim.x, c = C > 1 ? blockIdx.x % C : 0;
  const int lane = tid & 31, warp = tid >> 5, nw = T >> 5;
  for (int i = tid; i < N2; i += T) tw[i] = cvt<R>(a.twy[i]);
  ZRowLane<R, V> L;
  L.t = lane & 1;
  L.sg = L.t ? (R)-1 : (R)1;
  L.g = conjc(cvt<R>(a.twN[L.t]));
  pdl_wait();
  __syncthreads();
  const long long plane = (long long)(blockIdx.x / C) * a.nky * a.kzp;

  // y-inverse: entry n = j + R2 i, row k1 + R1 k2 in slot k1 R2 + k2
  for (int w = tid; w < a.nin * R2 * a.nkz; w += T) {
    const int fj = __umulhi(w, a.mkz), col = w - fj * a.nkz, j = fj % R2, f = fj / R2;
    const cx<R>* src = reinterpret_cast<const cx<R>*>(ps.src[f]) + plane + col;
    cx<R> v[R1];
#pragma unroll
    for (int i = 0; i < R1; ++i) {
      const int r = amap_row(a.ay, j + R2 * i);
      v[i] = r >= 0 ? src[r * a.kzp] : mkc<R>(0, 0);
    }
    DFT<R1, +1, R>::run(v);
    cx<R>* d = in + (f * NR + j) * a.rin + col;
#pragma unroll
    for (int k = 0; k < R1; ++k)
      if (C == 1 || k / KC == c) d[k % KC * R2 * a.rin] = k ? v[k] * conjc(tw[j * k]) : v[k];
  }
  __syncthreads();
  for (int w = tid; w < a.nin * KC * a.nkz; w += T) {
    const int fk = __umulhi(w, a.mkz), col = w - fk * a.nkz;
    cx<R>* d = in + fk * R2 * a.rin + col;
    cx<R> v[R2];
#pragma unroll
    for (int j = 0; j < R2; ++j) v[j] = d[j * a.rin];
    DFT<R2, +1, R>::run(v);
#pragma unroll
    for (int j = 0; j < R2; ++j) d[j * a.rin] = v[j];
  }
  __syncthreads();

  // c2r, a lane's value k in entry t + 2 k of its row
  for (int w = warp * 16; w < a.nin * NR; w += nw * 16) {
    const int r = w + (lane >> 1);
    const bool ok = r < a.nin * NR;
    cx<R>* row = in + (ok ? r : w) * a.rin + L.t;
    cx<R> x[V], v[V], xM = mkc<R>(0, 0);
#pragma unroll
    for (int j = 0; j < V; ++j) x[j] = (L.t + 2 * j < a.nkz) ? row[2 * j] : mkc<R>(0, 0);
    if (M < a.nkz && L.t == 0) xM = row[M];
    L.template pre<0>(x, xM, v);
    DFT<V, +1, R>::run(v);
    L.template lane_tws<+1, 1>(v);
    L.lane_bfly(v);
    __syncwarp();
    if (ok) {
#pragma unroll
      for (int k = 0; k < V; ++k) row[2 * k] = v[k];
    }
  }
  __syncthreads();
  // products and r2c
  const R sc = (R)a.scale, hs = (R)0.5 * sc;
  for (int w = warp * 16; w < a.nprod * NR; w += nw * 16) {
    const int qr = w + (lane >> 1);
    const bool ok = qr < a.nprod * NR;
    const int q = ok ? qr / NR : 0, fs = NR * a.rin;
    const cx<R>* row = in + qr % NR * a.rin + L.t;
    const cx<R>*xa = row + pp.a[q] * fs, *xb = row + pp.b[q] * fs;
    cx<R> v[V];
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = rmul(xa[2 * k], xb[2 * k]);
    if (pp.c[q] >= 0) {
      const cx<R>*xc = row + pp.c[q] * fs, *xd = row + pp.d[q] * fs;
#pragma unroll
      for (int k = 0; k < V; ++k) v[k] = v[k] - rmul(xc[2 * k], xd[2 * k]);
    }
    __syncwarp();
    L.lane_bfly(v);
    L.template lane_tws<-1, 1>(v);
    DFT<V, -1, R>::run(v);
    cx<R>* d = out + qr * a.rout;
    L.template post<0>(v, hs, d, ok ? a.nkz : 0);
    if (ok && L.t == 0 && a.nkz > M) d[M] = mkc<R>(sc * (v[0].x - v[0].y), (R)0);
  }
  __syncthreads();

  // y-forward, the adjoint
  for (int w = tid; w < a.nprod * KC * a.nkz; w += T) {
    const int qk = __umulhi(w, a.mkz), col = w - qk * a.nkz, k = qk % KC + c * KC;
    cx<R>* d = out + qk * R2 * a.rout + col;
    cx<R> v[R2];
#pragma unroll
    for (int j = 0; j < R2; ++j) v[j] = d[j * a.rout];
    DFT<R2, -1, R>::run(v);
    d[0] = v[0];
#pragma unroll
    for (int j = 1; j < R2; ++j) d[j * a.rout] = v[j] * tw[j * k];
  }
  if constexpr (C > 1) cg::this_cluster().sync();
  else __syncthreads();
  const cx<R>* part[C];
#pragma unroll
  for (int b = 0; b < C; ++b) part[b] = C > 1 ? cg::this_cluster().map_shared_rank(out, b) : out;
  for (int w = c * T + tid; w < a.nprod * R2 * a.kzp; w += C * T) {
    const int qj = __umulhi(w, a.mkzp), col = w - qj * a.kzp, j = qj % R2, q = qj / R2;
    const int o = (q * NR + j) * a.rout + col;
    cx<R>* dst = reinterpret_cast<cx<R>*>(ps.dst[q]) + plane + col;
    cx<R> v[R1];
#pragma unroll
    for (int k = 0; k < R1; ++k) v[k] = col < a.nkz ? part[k / KC][o + k % KC * R2 * a.rout] : mkc<R>(0, 0);
    DFT<R1, -1, R>::run(v);
#pragma unroll
    for (int i = 0; i < R1; ++i) {
      const int r = amap_row(a.ay, j + R2 * i);
      if (r >= 0) dst[r * a.kzp] = v[i];
    }
  }
  if constexpr (C > 1) cg::this_cluster().sync();  // the others may still read this block's slots
}

// the least stride of n entries or more that is 2 modulo 4
int row_stride(int n) { return n + ((2 - n % 4) + 4) % 4; }

int in_stride(const PlaneLaunch& l) { return row_stride(l.M > l.a.nkz ? l.M : l.a.nkz); }
// m with __umulhi(w, m) = w / n for every w < 2^16, 1 < n < 2^16
unsigned reciprocal(int n) { return (unsigned)((1ull << 32) / n + 1); }

size_t plane_smem(const PlaneLaunch& l, int C) {
  const size_t esz = l.prec == F64 ? 16 : 8;
  return esz * (l.N2 + l.N2 / C * ((size_t)l.a.nin * in_stride(l) + (size_t)l.a.nprod * row_stride(l.a.nkz)));
}

// two blocks a plane where the planes leave half the chip idle and one block would go over the products' rows
// with more than ten warps
int plane_blocks(const PlaneLaunch& l) { return l.nplanes * 2 <= 148 && l.a.nprod * l.N2 > 160 ? 2 : 1; }

template <typename R, int R1, int R2, int V, int C>
cudaError_t run_plane_c(const PlaneLaunch& l, cudaStream_t s) {
  auto kern = k_plane<R, R1, R2, V, C>;
  const size_t smem = plane_smem(l, C);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e != cudaSuccess) return e;
  // as many warps as the products' rows take; two blocks an SM where there are that many
  const bool two = l.nplanes * C > 148 && 2 * smem <= kPlaneSmem;
  const int T = std::min(32 * ((l.a.nprod * (l.N2 / C) + 15) / 16), two ? 320 : PlaneThreads<R>::v);
  cudaLaunchAttribute attr[2]{};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = C;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(l.nplanes * C));
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = C > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, l.a, l.ps, l.pp);
}

template <typename R, int R1, int R2, int V>
cudaError_t run_plane(const PlaneLaunch& l, cudaStream_t s) {
  return plane_blocks(l) == 2 ? run_plane_c<R, R1, R2, V, 2>(l, s) : run_plane_c<R, R1, R2, V, 1>(l, s);
}

template <typename R>
cudaError_t run_plane_n(const PlaneLaunch& l, cudaStream_t s) {
  if (l.M == 16) return l.N2 == 32 ? run_plane<R, 8, 4, 8>(l, s) : run_plane<R, 8, 8, 8>(l, s);
  return l.N2 == 32 ? run_plane<R, 8, 4, 16>(l, s) : run_plane<R, 8, 8, 16>(l, s);
}

}  // namespace

// The lines: a block's time does not fall with the number of planes, the three passes' does.  Steps measured
// (this form / the three passes, us): planes of 32 x 32 gain whatever their number (FP32 fluid with 4 of them
// 51.0 / 57.6, with 16 55.5 / 63.7; FP64 MHD with 6 75.9 / 80.0, with 16 69.8 / 76.3).  Larger ones: 64 x 64 FP64 fluid 86 / 78 with 16 or 32 planes, 111 / 112 with 48, 90.6 / 96.3
// with 64 (two blocks each, to 74), 146 / 148 with 80, 148 / 158 with 96, 128 / 150 with 128, 226 / 258 with 256;
// FP32 fluid 71 / 68, 96 / 100, 76 / 81, 120 / 119, 123 / 125, 103 / 113, 146 / 179; FP32 MHD 88 / 80, 115 / 117,
// 98 / 98, 150 / 154, 154 / 162, - , 255 / 292; 64 x 32 FP32 MHD 74 / 84 with 64 planes, 150 / 204 with 256;
// 32 x 64 FP64 scalar 86 / 88 and 206 / 249.  A plane has to fit one block: two a plane over more than one wave
// lost (64 x 64 FP64 MHD 508 / 477 with 256 planes).
// Looks at one request's geometry only, so a batched request takes the path of a lone one; the number of blocks
// that share a plane follows the batch, but changes no operation.
bool plane_fits(const PlaneLaunch& l, int N1) {
  if ((l.N2 != 32 && l.N2 != 64) || (l.M != 16 && l.M != 32) || l.a.nkz < 2) return false;
  if (plane_smem(l, 1) > kPlaneSmem || l.nplanes >= (1LL << 29)) return false;
  return l.N2 * l.M <= 512 || (N1 >= 48 && N1 <= 74) || N1 >= 96;
}

cudaError_t launch_plane(PlaneLaunch l, cudaStream_t s) {
  l.a.rin = in_stride(l);
  l.a.rout = row_stride(l.a.nkz);
  l.a.mkz = reciprocal(l.a.nkz);
  l.a.mkzp = reciprocal(l.a.kzp);
  return l.prec == F64 ? run_plane_n<double>(l, s) : run_plane_n<float>(l, s);
}

}  // namespace tg
