// Dispatch of the strided-axis c2c kernels (x- and y-passes).
//
// Power-of-two lengths 16..256 whose stored input and kept output rows fit one TMA box (<= 256
// rows) run k_axis_tma: the block's column tile moves HBM -> shared memory and back as single
// tiled bulk tensor copies, so the threads spend no instructions on addresses or row maps of
// global memory.  Power-of-two lengths beyond that run the register-staged k_axis_c2c, every
// other length the mixed-radix k_axis_mixed, or the direct sum k_axis_dft where that is faster.
// k_axis_tma and k_axis_c2c compute the same butterflies in the same order (equal results up to
// how the compiler contracts multiply-adds in each kernel).
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "tg_fft_dmma.cuh"
#include "tg_fft_fold.cuh"
#include "tg_fft_launch.h"
#include "tg_fft_mixed.cuh"
#include "tg_fft_tc.cuh"
#include "tg_tma.cuh"

namespace tg {

bool axis_tma_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("TG_AXIS_TMA");
    return !(e && e[0] == '0');
  }();
  return on;
}

namespace {

// set by a TMA-staged block whose tile never arrived within the bounded wait
__device__ int g_axis_tma_timeout = 0;

constexpr int kTmaPolls = 1 << 20;

struct TmaSet {
  CUtensorMap src[kMaxPtr];
  CUtensorMap src2[kMaxPtr];
  CUtensorMap dst[kMaxPtr];
};

// One block: W columns (TmaW) of one batch of one field.  Tile rows in shared memory are
// row-major [row][W]; the same buffer holds the loaded input tile, then the transposed
// intermediate, then the output tile.
// Tile width of the TMA axis kernel: 8 columns (64 or 128 contiguous bytes per row), so the
// solver's column counts (kzp, a multiple of 8, and nky * kzp) split into whole tiles; the block
// has W * R1 threads (128 at L = 256).  (16-column FP32 tiles, 128-byte row segments at 256
// threads a block, measured no faster: 256^3 FP32-mixed step 1.85 ms against 1.81 ms.)
template <typename Rw>
struct TmaW {
  static constexpr int v = 8;
};
// resident blocks per SM the kernel is built for: 64 registers (FP32 arithmetic) or 80 (FP64)
template <typename Rw, int NT>
struct AxisOcc {
  static constexpr int v = (65536 / NT) / (sizeof(Rw) == 4 ? 64 : 80);
};

template <typename Ri, typename Ro, typename Rw, int R1, int R2, int DIR, bool COMB>
__global__ void __launch_bounds__(TmaW<Rw>::v * R1, AxisOcc<Rw, TmaW<Rw>::v * R1>::v)
    k_axis_tma(AxisArgs a, const __grid_constant__ TmaSet tm, int nin_rows, int nout_rows, unsigned tile_bytes) {
  constexpr int L = R1 * R2;
  constexpr int W = TmaW<Rw>::v;
  constexpr int NT = W * R1;
  constexpr int CEi = (int)(sizeof(cx<Ri>) / 8), CEo = (int)(sizeof(cx<Ro>) / 8);
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  uint64_t* bar = reinterpret_cast<uint64_t*>(base);
  int* ok_flag = reinterpret_cast<int*>(base + 8);
  cx<Rw>* tw = reinterpret_cast<cx<Rw>*>(base + 128);
  unsigned char* buf = base + 128 + ((L * sizeof(cx<Rw>) + 127) & ~(size_t)127);
  unsigned char* buf2 = buf + tile_bytes;
  const int tid = threadIdx.x;
  const int f = blockIdx.z, b = blockIdx.y, col0 = blockIdx.x * W;
  if (tid == 0) {
    mbar_init(bar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  pdl_wait();
  if (tid == 0) {
    const unsigned in_bytes = (unsigned)(W * CEi * 8) * (unsigned)nin_rows;
    mbar_arrive_expect_tx(bar, COMB ? 2 * in_bytes : in_bytes);
    tma_load_3d(buf, &tm.src[f], col0 * CEi, 0, b, bar);
    if constexpr (COMB) tma_load_3d(buf2, &tm.src2[f], col0 * CEi, 0, b, bar);
  }
  for (int i = tid; i < L; i += NT) {
    cx<Rw> t = cvt<Rw>(a.tw[i]);
    if (DIR > 0) t.y = -t.y;
    tw[i] = t;
  }
  if (tid == 0) {
    const bool ok = mbar_wait_bounded(bar, 0, a.wait_short ? 0 : kTmaPolls);
    *ok_flag = ok ? 1 : 0;
    if (!ok) {
      atomicExch(a.wait_flag ? a.wait_flag : &g_axis_tma_timeout, 1);
      mbar_wait_bounded(bar, 0, kTmaPolls);  // let a late copy land before the block leaves
    }
  }
  __syncthreads();
  if (*ok_flag == 0) return;
  mbar_wait_bounded(bar, 0, 64);  // the phase has completed: acquire the copied tile
  const int w = tid % W;
  const int n2 = tid / W;
  cx<Rw> v[R1];
  if (n2 < R2) {
    const cx<Ri>* tin = reinterpret_cast<const cx<Ri>*>(buf);
    const cx<Ri>* tin2 = reinterpret_cast<const cx<Ri>*>(buf2);
    const int comb = COMB ? a.comb[f] : 0;
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) {
      const int r = amap_row(a.in, R2 * n1 + n2);
      v[n1] = mkc<Rw>(0, 0);
      if (r >= 0) {
        v[n1] = cvt<Rw>(tin[r * W + w]);
        if constexpr (COMB) {
          if (comb > 0) v[n1] = v[n1] + cvt<Rw>(tin2[r * W + w]);
          else if (comb < 0) v[n1] = v[n1] - cvt<Rw>(tin2[r * W + w]);
        }
      }
    }
    DFT<R1, DIR, Rw>::run(v);
  }
  __syncthreads();  // the input tile is consumed; its buffer takes the intermediate
  cx<Rw>* ex = reinterpret_cast<cx<Rw>*>(buf);
  if (n2 < R2) {
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) ex[(k1 * R2 + n2) * W + w] = v[k1] * tw[(n2 * k1) & (L - 1)];
  }
  __syncthreads();
  const int k1 = tid / W;
  cx<Rw> u[R2];
#pragma unroll
  for (int m = 0; m < R2; ++m) u[m] = ex[(k1 * R2 + m) * W + w];
  DFT<R2, DIR, Rw>::run(u);
  __syncthreads();  // the intermediate is consumed; the buffer takes the output tile
  cx<Ro>* tout = reinterpret_cast<cx<Ro>*>(buf);
  const Rw sc = (Rw)a.scale;
#pragma unroll
  for (int k2 = 0; k2 < R2; ++k2) {
    const int r = amap_row(a.out, k1 + R1 * k2);
    if (r >= 0) tout[r * W + w] = cvt<Ro>(sc * u[k2]);
  }
  fence_proxy_async_smem();
  __syncthreads();
  if (tid == 0) {
    tma_store_3d(&tm.dst[f], col0 * CEo, 0, b, buf);
    bulk_commit_group();
    bulk_wait_group_read0();
  }
}

template <typename Ri, typename Ro, typename Rw, int R1, int R2, int DIR>
cudaError_t run_axis_tma(const AxisLaunch& l, cudaStream_t s, bool* used) {
  *used = false;
  constexpr int L = R1 * R2;
  constexpr int W = TmaW<Rw>::v;
  constexpr int NT = W * R1;
  constexpr int CEi = (int)(sizeof(cx<Ri>) / 8), CEo = (int)(sizeof(cx<Ro>) / 8);
  const int nin_rows = amap_count(l.a.in), nout_rows = amap_count(l.a.out);
  if (nin_rows < 1 || nin_rows > 256 || nout_rows < 1 || nout_rows > 256) return cudaSuccess;
  if (l.nbatch > 65535) return cudaSuccess;
  bool comb = false;
  for (int f = 0; f < l.nfields; ++f) comb = comb || (l.a.comb[f] != 0);
  TmaSet tm;  // host staging of the maps (copied into the launch parameters)
  std::memset(&tm, 0, sizeof(tm));
  for (int f = 0; f < l.nfields; ++f) {
    if (!tma_map_3d(&tm.src[f], l.ps.src[f], (unsigned long long)l.a.ncols * CEi, (unsigned long long)nin_rows,
                    (unsigned long long)l.nbatch, (unsigned long long)l.a.sr * sizeof(cx<Ri>),
                    (unsigned long long)l.a.sb * sizeof(cx<Ri>), W * CEi, nin_rows))
      return cudaSuccess;
    if (comb && l.a.comb[f] != 0 &&
        !tma_map_3d(&tm.src2[f], l.ps.src2[f], (unsigned long long)l.a.ncols * CEi, (unsigned long long)nin_rows,
                    (unsigned long long)l.nbatch, (unsigned long long)l.a.sr * sizeof(cx<Ri>),
                    (unsigned long long)l.a.sb * sizeof(cx<Ri>), W * CEi, nin_rows))
      return cudaSuccess;
    if (comb && l.a.comb[f] == 0) tm.src2[f] = tm.src[f];
    if (!tma_map_3d(&tm.dst[f], l.ps.dst[f], (unsigned long long)l.a.ncols * CEo, (unsigned long long)nout_rows,
                    (unsigned long long)l.nbatch, (unsigned long long)l.a.dr * sizeof(cx<Ro>),
                    (unsigned long long)l.a.db * sizeof(cx<Ro>), W * CEo, nout_rows))
      return cudaSuccess;
  }
  size_t tile = (size_t)W * nin_rows * sizeof(cx<Ri>);
  tile = tile > (size_t)W * L * sizeof(cx<Rw>) ? tile : (size_t)W * L * sizeof(cx<Rw>);
  tile = tile > (size_t)W * nout_rows * sizeof(cx<Ro>) ? tile : (size_t)W * nout_rows * sizeof(cx<Ro>);
  tile = (tile + 127) & ~(size_t)127;
  const size_t smem = 128 + 128 + ((L * sizeof(cx<Rw>) + 127) & ~(size_t)127) + tile +
                      (comb ? (size_t)W * nin_rows * sizeof(cx<Ri>) : 0);
  if (smem > 200 * 1024) return cudaSuccess;
  dim3 grid((l.a.ncols + W - 1) / W, l.nbatch, l.nfields);
  cudaError_t e;
  if (comb) {
    auto kern = k_axis_tma<Ri, Ro, Rw, R1, R2, DIR, true>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return e;
    e = launch_pdl(kern, grid, NT, smem, s, l.a, tm, nin_rows, nout_rows, (unsigned)tile);
  } else {
    auto kern = k_axis_tma<Ri, Ro, Rw, R1, R2, DIR, false>;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return e;
    e = launch_pdl(kern, grid, NT, smem, s, l.a, tm, nin_rows, nout_rows, (unsigned)tile);
  }
  *used = true;
  return e;
}

template <typename Ri, typename Ro, typename Rw, int R1, int R2, int DIR>
cudaError_t run_axis_fast(const AxisLaunch& l, cudaStream_t s) {
  constexpr int L = R1 * R2;
  constexpr int W = 256 / R1;
  if constexpr (L >= 16 && L <= 256) {
    if (axis_tma_enabled()) {
      bool used = false;
      cudaError_t e = run_axis_tma<Ri, Ro, Rw, R1, R2, DIR>(l, s, &used);
      if (e != cudaSuccess || used) return e;
    }
  }
  const size_t smem = (size_t)(L + (size_t)L * W) * sizeof(cx<Rw>);
  auto kern = k_axis_c2c<Ri, Ro, Rw, R1, R2, DIR>;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  dim3 grid((l.a.ncols + W - 1) / W, l.nbatch, l.nfields);
  return launch_pdl(kern, grid, 256, smem, s, l.a, l.ps);
}

// lengths that are no power of two (or beyond the register-staged kernels): the mixed-radix
// Stockham pass.  Eight columns a tile while two tiles fit beside another block's, else four, two
// or one.  Threads: what the stage of most butterflies has work for, at most kMixThreads.
template <typename Ri, typename Ro, typename Rw, int DIR>
cudaError_t run_axis_mixed(const AxisLaunch& l, cudaStream_t s) {
  MixPlan p;
  if (!mix_plan(l.L, p)) return cudaErrorInvalidValue;
  auto bytes = [&](int w) { return (size_t)(l.L + ((size_t)l.L << (w + 1))) * sizeof(cx<Rw>); };
  while (p.wsh > 0 && bytes(p.wsh) > 100 * 1024) --p.wsh;
  const size_t smem = bytes(p.wsh);
  if (smem > 227 * 1024) return cudaErrorInvalidValue;
  int threads = 32;
  for (int i = 0; i < p.ns; ++i) {
    const int items = mix_reg_radix(p.r[i]) ? (l.L / p.r[i]) << p.wsh : l.L << p.wsh;
    threads = std::max(threads, std::min(kMixThreads, (items + 31) / 32 * 32));
  }
  const int W = 1 << p.wsh;
  auto kern = k_axis_mixed<Ri, Ro, Rw, DIR>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((l.a.ncols + W - 1) / W, l.nbatch, l.nfields);
  e = launch_pdl(kern, grid, threads, smem, s, l.a, l.ps, p);
  return e;
}

// The launches of the direct sum (k_axis_dft) among those of no power of two.  Measured in a chain of launches
// (B200, us, direct / mixed-radix, FP64):
//  * a prime factor of 11 and more, up to 26, any size: 4 x 4096 columns of 13 6.0 / 8.2, 23 8.7 / 10.9, 26 10.3 / 11.4
//    (29 12.4 / 12.4, 34 17.1 / 15.6); 4 x 256 columns 2.0 / 2.5, 2.4 / 3.0, 2.5 / 3.0;
//  * up to 14 where one request has two blocks an SM or less, a chain of latencies: 4 x 256 columns of 6 1.8 / 2.7, 10
//    1.9 / 3.4, 12 2.0 / 3.7; larger requests go the other way (4 x 2048 columns 3.2 / 3.0, 3.8 / 3.7, 4.0 / 4.0).
//    From 15 on a lone request gains as well (20 x 24 x 32 MHD FP32-mixed step 82 / 98), but a batch, which takes a lone
//    request's path, loses more than a tenth (64 requests 844 / 711).
constexpr int kDftMaxPrime = 26, kDftMax = 14;
constexpr long long kDftMaxBlocks = 2 * 148;
bool dft_taken(const AxisLaunch& l) {
  int m = l.L;
  for (int q : {2, 3, 5, 7})
    while (m % q == 0) m /= q;
  if (m > 1) return l.L <= kDftMaxPrime;
  const long long blocks = (long long)((l.a.ncols + kDftCols - 1) / kDftCols) * (l.nbatch / l.nreq) * l.nfields;
  return l.L <= kDftMax && blocks <= kDftMaxBlocks;
}
template <typename Ri, typename Ro, typename Rw, int DIR>
cudaError_t run_axis_dft(const AxisLaunch& l, cudaStream_t s) {
  const size_t smem = (size_t)l.L * (1 + kDftCols) * sizeof(cx<Rw>);  // 3.7 KB at most
  dim3 grid((l.a.ncols + kDftCols - 1) / kDftCols, l.nbatch, l.nfields);
  return launch_pdl(k_axis_dft<Ri, Ro, Rw, DIR>, grid, kDftThreads, smem, s, l.a, l.ps, l.L);
}

template <typename Ri, typename Ro, typename Rw, int DIR>
cudaError_t run_axis_dir(const AxisLaunch& l, cudaStream_t s) {
  switch (l.L) {
    case 2: return run_axis_fast<Ri, Ro, Rw, 2, 1, DIR>(l, s);
    case 4: return run_axis_fast<Ri, Ro, Rw, 2, 2, DIR>(l, s);
    case 8: return run_axis_fast<Ri, Ro, Rw, 4, 2, DIR>(l, s);
    case 16: return run_axis_fast<Ri, Ro, Rw, 4, 4, DIR>(l, s);
    case 32: return run_axis_fast<Ri, Ro, Rw, 8, 4, DIR>(l, s);
    case 64: return run_axis_fast<Ri, Ro, Rw, 8, 8, DIR>(l, s);
    case 128: return run_axis_fast<Ri, Ro, Rw, 16, 8, DIR>(l, s);
    case 256: return run_axis_fast<Ri, Ro, Rw, 16, 16, DIR>(l, s);
    case 512: return run_axis_fast<Ri, Ro, Rw, 32, 16, DIR>(l, s);
    default:
      if (l.L < 1 || l.L > 2048) return cudaErrorInvalidValue;
      if (dft_taken(l)) return run_axis_dft<Ri, Ro, Rw, DIR>(l, s);
      return run_axis_mixed<Ri, Ro, Rw, DIR>(l, s);
  }
}

template <typename Ri, typename Ro, typename Rw>
cudaError_t run_axis_prec(const AxisLaunch& l, cudaStream_t s) {
  return l.dir < 0 ? run_axis_dir<Ri, Ro, Rw, -1>(l, s) : run_axis_dir<Ri, Ro, Rw, +1>(l, s);
}

// the matrix-product x-pass when every field's kind has its matrix and the tiles fit
template <typename Ri, typename Ro, typename Rw>
cudaError_t run_r2r_mm(const AxisLaunch& l, const R2RArgs& r, cudaStream_t s, bool* used) {
  *used = false;
  const int nin = amap_count(l.a.in);
  int rpad = 0;
  for (int f = 0; f < l.nfields; ++f) {
    const int k = r.kind[f];
    if (k < 0 || k > 3 || !r.mat[k] || r.mat_rows[k] != amap_count(l.a.out) || r.mat_cols[k] != nin)
      return cudaSuccess;
    rpad = std::max(rpad, (r.mat_rows[k] + 31) / 32 * 32);
  }
  // 64-column tiles when they fit in shared memory, else 32
  int cw = 64;
  size_t smem = (size_t)nin * cw * sizeof(cx<Rw>) + (size_t)nin * rpad * sizeof(Rw);
  if (smem > 200 * 1024) {
    cw = 32;
    smem = (size_t)nin * cw * sizeof(cx<Rw>) + (size_t)nin * rpad * sizeof(Rw);
  }
  if (smem > 200 * 1024) return cudaSuccess;
  auto kern = cw == 64 ? k_axis_r2r_mm<Ri, Ro, Rw, 64> : k_axis_r2r_mm<Ri, Ro, Rw, 32>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((l.a.ncols + cw - 1) / cw, l.nbatch, l.nfields);
  e = launch_pdl(kern, grid, 256, smem, s, l.a, l.ps, r);
  *used = true;
  return e;
}

// the folded register-tiled matrix product (k_axis_r2r_fold) unless TG_R2R_GEMM=0
bool r2r_gemm_enabled() {
  static const bool on = [] {
    const char* e = std::getenv("TG_R2R_GEMM");
    return !(e && e[0] == '0');
  }();
  return on;
}

// every field's kind has its matrix (all of the same size and direction) and the launch maps all N
// points to the stored coefficients or back
bool r2r_foldable(const AxisLaunch& l, const R2RArgs& r, bool& fwd) {
  if (!r2r_gemm_enabled()) return false;
  const int nin = amap_count(l.a.in), nout = amap_count(l.a.out);
  fwd = r.kind[0] <= 1;
  for (int f = 0; f < l.nfields; ++f) {
    const int k = r.kind[f];
    if (k < 0 || k > 3 || (k <= 1) != fwd || !r.mat[k] || r.mat_rows[k] != nout || r.mat_cols[k] != nin || l.a.comb[f])
      return false;
  }
  return (fwd ? nin : nout) == l.L && nin >= 1 && nout >= 1;
}

template <typename Ri, int RT, bool FWD>
cudaError_t run_r2r_fold_rt(const AxisLaunch& l, const R2RArgs& r, int ntile, int steps, cudaStream_t s) {
  const size_t smem = (size_t)kFoldAhead * 2 * kFoldCols * sizeof(cx<Ri>) +
                      (size_t)steps * ((RT + 3) / 4 * 8) * sizeof(float);
  auto kern = k_axis_r2r_fold<Ri, RT, FWD>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e != cudaSuccess) return e;
  dim3 grid((l.a.ncols + kFoldCols - 1) / kFoldCols, l.nbatch, l.nfields * ntile);
  e = launch_pdl(kern, grid, kFoldThreads, smem, s, l.a, l.ps, r, l.L, ntile);
  return e;
}

// FP32: row tiles of 22 pairs, or of 11 where those leave an SM without its two blocks (every tile
// reads the inputs again, so the larger one where the grid allows)
template <typename Ri>
cudaError_t run_r2r_fold(const AxisLaunch& l, const R2RArgs& r, cudaStream_t s, bool* used) {
  *used = false;
  bool fwd;
  if (!r2r_foldable(l, r, fwd)) return cudaSuccess;
  const int nin = amap_count(l.a.in), nout = amap_count(l.a.out), N = l.L;
  const int pairs = fwd ? (nout + 1) / 2 : (N + 1) / 2, steps = fwd ? (N + 1) / 2 : (nin + 1) / 2;
  const long long blocks = (long long)((l.a.ncols + kFoldCols - 1) / kFoldCols) * l.nbatch * l.nfields * ((pairs + 21) / 22);
  const int rt = blocks < 2 * 148 ? 11 : 22, ntile = (pairs + rt - 1) / rt;
  // 16-byte accesses of a thread's two columns: even column counts and strides (whole rows of kzp, a multiple of 8,
  // on every caller) and aligned buffers
  if (((l.a.ncols | l.a.sr | l.a.dr | l.a.sb | l.a.db) & 1) != 0) return cudaSuccess;
  for (int f = 0; f < l.nfields; ++f)
    if (((reinterpret_cast<uintptr_t>(l.ps.src[f]) | reinterpret_cast<uintptr_t>(l.ps.dst[f])) & 15) != 0) return cudaSuccess;
  if ((long long)l.nfields * ntile > 65535 || (size_t)steps * 48 * sizeof(float) > 96 * 1024) return cudaSuccess;
  *used = true;
  if (rt == 22)
    return fwd ? run_r2r_fold_rt<Ri, 22, true>(l, r, ntile, steps, s)
               : run_r2r_fold_rt<Ri, 22, false>(l, r, ntile, steps, s);
  return fwd ? run_r2r_fold_rt<Ri, 11, true>(l, r, ntile, steps, s)
             : run_r2r_fold_rt<Ri, 11, false>(l, r, ntile, steps, s);
}

// shared memory of k_axis_r2r_dmma: the ring of input stages and the block's coefficients
size_t dmma_smem(int mt, int nst) {
  return sizeof(double) * ((size_t)kDmStages * kDmStageD + (size_t)nst * (kDmPairs / 4) * 2 * mt * 32);
}

template <int MT, bool FWD>
cudaError_t run_r2r_dmma_mt(const AxisLaunch& l, const R2RArgs& r, int nrb, int nst, cudaStream_t s) {
  const size_t smem = dmma_smem(MT, nst);
  auto kern = k_axis_r2r_dmma<MT, FWD>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int ntiles = (l.a.ncols + kDmCols - 1) / kDmCols;
  const long long per = (long long)l.nbatch * l.nfields * nrb;
  const int P = (int)std::max<long long>(1, std::min<long long>(ntiles, 148 / per));
  dim3 grid(P, l.nbatch, l.nfields * nrb);
  e = launch_pdl(kern, grid, kDmThreads, smem, s, l.a, l.ps, r, l.L, nrb);
  return e;
}

// FP64: the folded product on the matrix instructions.  Row tiles of 8 MT pairs with MT the smaller
// of the two larger values if that needs no more row blocks (N1 = 129, 128: 6 forward, 9 inverse in
// one block; N1 = 65: 3 and 5), and the next smaller one while the coefficients of a block's rows do
// not fit beside the ring: MT = 2 fits every N1 of launch_r2r (196 KB at 1024).  Measured convection
// steps against the register-tiled product of the full matrix (us): N1 x 16 x 32 with N1 = 417 309 / 869,
// 513 451 / 1354; all modes stored 404 639 / 1659, 600 1320 / 4868.
cudaError_t run_r2r_dmma(const AxisLaunch& l, const R2RArgs& r, cudaStream_t s, bool* used) {
  *used = false;
  bool fwd;
  if (!r2r_foldable(l, r, fwd)) return cudaSuccess;
  const int nin = amap_count(l.a.in), nout = amap_count(l.a.out), N = l.L;
  for (int f = 0; f < l.nfields; ++f)  // 16-byte copies
    if (((reinterpret_cast<uintptr_t>(l.ps.src[f]) | reinterpret_cast<uintptr_t>(l.ps.dst[f])) & 15) != 0) return cudaSuccess;
  const int pairs = fwd ? (nout + 1) / 2 : (N + 1) / 2, mts = (pairs + 7) / 8;
  const int nst = ((fwd ? (N + 1) / 2 : (nin + 1) / 2) + kDmPairs - 1) / kDmPairs;
  const int tile[3] = {fwd ? 6 : 9, fwd ? 3 : 5, 2};
  int t = (mts + tile[1] - 1) / tile[1] <= (mts + tile[0] - 1) / tile[0] ? 1 : 0;
  while (t < 3 && dmma_smem(tile[t], nst) > 227 * 1024) ++t;
  if (t == 3) return cudaSuccess;
  const int nrb = (mts + tile[t] - 1) / tile[t];
  if ((long long)l.nfields * nrb > 65535) return cudaSuccess;
  *used = true;
  if (t == 2) return fwd ? run_r2r_dmma_mt<2, true>(l, r, nrb, nst, s) : run_r2r_dmma_mt<2, false>(l, r, nrb, nst, s);
  if (fwd) return t == 1 ? run_r2r_dmma_mt<3, true>(l, r, nrb, nst, s) : run_r2r_dmma_mt<6, true>(l, r, nrb, nst, s);
  return t == 1 ? run_r2r_dmma_mt<5, false>(l, r, nrb, nst, s) : run_r2r_dmma_mt<9, false>(l, r, nrb, nst, s);
}

// FP32 forms: the x-inverse contraction on the tensor cores (k_axis_r2r_tc, 3xTF32) when a field of
// one request spans at least kTcMinTiles column tiles (the per-block set-up, coefficient pairs and
// tensor memory, amortises) and the folded product needs more than kTcMinPairs row pairs, three row
// tiles of 22 that each read the inputs again.  Measured launches, tensor cores against folded:
// inverse 129 x 256 x 256 56.4 / 70.1 us, 97 x 128 x 256 30.0 / 38.6, 65 x 256 x 128 23.7 / 20.1,
// 65 x 128 x 128 19.4 / 17.1; forward 133.7 / 115.1, 54.0 / 52.0, 40.5 / 26.7, 26.1 / 16.6.  The rule
// looks at one request's geometry only, so a request batched in the serving loop takes the same path
// as on a lone context.  TG_R2R_TC=0 never, =1 always.
constexpr int kTcMinTiles = 16;
constexpr int kTcMinPairs = 45;
int r2r_tc_mode() {
  static const int m = [] {
    const char* e = std::getenv("TG_R2R_TC");
    if (e && e[0] == '0') return 0;
    if (e && e[0] == '1') return 1;
    return 2;
  }();
  return m;
}

template <typename Ri>
cudaError_t run_r2r_tc(const AxisLaunch& l, const R2RArgs& r, cudaStream_t s, bool* used) {
  *used = false;
  const int mode = r2r_tc_mode();
  if (mode == 0) return cudaSuccess;
  if (mode == 2 && ((2LL * l.a.ncols + 127) / 128 < kTcMinTiles || r.kind[0] <= 1 || (l.L + 1) / 2 < kTcMinPairs))
    return cudaSuccess;
  const int nin = amap_count(l.a.in), nout = amap_count(l.a.out);
  for (int f = 0; f < l.nfields; ++f) {
    const int k = r.kind[f];
    if (k < 0 || k > 3 || !r.mat[k] || r.mat_rows[k] != nout || r.mat_cols[k] != nin) return cudaSuccess;
    if (l.a.comb[f]) return cudaSuccess;
  }
  if (nin < 1 || nout < 1) return cudaSuccess;
  TcArgs t{};
  t.npad = (nout + 15) / 16 * 16;
  t.kpad = (nin + 7) / 8 * 8;
  if (t.npad > 256) return cudaSuccess;
  t.tmem_cols = 32;  // per accumulator; two of them
  while (t.tmem_cols < t.npad) t.tmem_cols *= 2;
  t.ntiles = (int)((2LL * l.a.ncols + 127) / 128);
  // coefficient pairs, nab operand slots of [hi, lo] chunks, eleven mbarriers, slot and flag;
  // three slots where they fit
  auto bytes = [&](int nab) {
    return sizeof(float) * (2 * (size_t)t.npad * t.kpad + 2 * (size_t)nab * 128 * kTcKC) +
           sizeof(uint64_t) * (2 * kTcMaxNab + 5) + 16;
  };
  int nab = kTcMaxNab;
  while (nab > 1 && bytes(nab) > 227 * 1024) --nab;
  const size_t smem = bytes(nab);
  if (smem > 227 * 1024) return cudaSuccess;
  t.nab = nab;
  auto kern = k_axis_r2r_tc<Ri>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  // one block per SM (shared memory, tensor memory): one persistent wave of at most 148 blocks,
  // or one block per (batch, field) when those alone exceed it
  const int per = l.nbatch * l.nfields;
  const int P = std::max(1, std::min(t.ntiles, 148 / per));
  *used = true;
  dim3 grid(P, l.nbatch, l.nfields);
  e = launch_pdl(kern, grid, kTcThreads, smem, s, l.a, l.ps, r, t);
  return e;
}

template <typename Ri, typename Ro, typename Rw>
cudaError_t run_r2r(const AxisLaunch& l, const R2RArgs& r, int N, cudaStream_t s) {
  if constexpr (sizeof(Ro) == 4 && sizeof(Rw) == 4) {
    bool used = false;
    cudaError_t e = run_r2r_tc<Ri>(l, r, s, &used);
    if (e != cudaSuccess || used) return e;
  }
  if constexpr (sizeof(Rw) == 8) {
    bool used = false;
    cudaError_t e = run_r2r_dmma(l, r, s, &used);
    if (e != cudaSuccess || used) return e;
  }
  if constexpr (sizeof(Ro) == 4 && sizeof(Rw) == 4) {
    bool used = false;
    cudaError_t e = run_r2r_fold<Ri>(l, r, s, &used);
    if (e != cudaSuccess || used) return e;
  }
  {
    bool used = false;
    cudaError_t e = run_r2r_mm<Ri, Ro, Rw>(l, r, s, &used);
    if (e != cudaSuccess || used) return e;
  }
  const int nin = amap_count(l.a.in);
  const size_t smem = (size_t)(4 * N + (size_t)nin * 32) * sizeof(cx<Rw>);
  auto kern = k_axis_r2r<Ri, Ro, Rw>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((l.a.ncols + 31) / 32, l.nbatch, l.nfields);
  e = launch_pdl(kern, grid, 256, smem, s, l.a, l.ps, r, N);
  return e;
}

}  // namespace

cudaError_t launch_r2r(const AxisLaunch& l, const R2RArgs& r, cudaStream_t s) {
  if (l.a.ncols <= 0 || l.nbatch <= 0 || l.nfields <= 0) return cudaSuccess;
  if (l.nbatch > 65535 || l.nfields > kMaxPtr || l.L < 2 || l.L > 1024) return cudaErrorInvalidValue;
  const int N = l.L;
  if (l.pwork == F64) {
    if (l.pin == F64 && l.pout == F64) return run_r2r<double, double, double>(l, r, N, s);
    return cudaErrorInvalidValue;
  }
  if (l.pin == F64 && l.pout == F64) return run_r2r<double, double, float>(l, r, N, s);
  if (l.pin == F64 && l.pout == F32) return run_r2r<double, float, float>(l, r, N, s);
  if (l.pin == F32 && l.pout == F32) return run_r2r<float, float, float>(l, r, N, s);
  if (l.pin == F32 && l.pout == F64) return run_r2r<float, double, float>(l, r, N, s);
  return cudaErrorInvalidValue;
}

cudaError_t launch_axis(const AxisLaunch& l, cudaStream_t s) {
  if (l.a.ncols <= 0 || l.nbatch <= 0 || l.nfields <= 0) return cudaSuccess;
  if (l.nbatch > 65535 || l.nfields > kMaxPtr) return cudaErrorInvalidValue;
  if (l.pwork == F64) {
    if (l.pin == F64 && l.pout == F64) return run_axis_prec<double, double, double>(l, s);
    return cudaErrorInvalidValue;
  }
  if (l.pin == F64 && l.pout == F64) return run_axis_prec<double, double, float>(l, s);
  if (l.pin == F64 && l.pout == F32) return run_axis_prec<double, float, float>(l, s);
  if (l.pin == F32 && l.pout == F32) return run_axis_prec<float, float, float>(l, s);
  if (l.pin == F32 && l.pout == F64) return run_axis_prec<float, double, float>(l, s);
  return cudaErrorInvalidValue;
}

int axis_tma_timeout(bool clear) {
  int h = 0;
  if (cudaMemcpyFromSymbol(&h, g_axis_tma_timeout, sizeof(int)) != cudaSuccess) return -1;
  if (clear && h) {
    const int z = 0;
    cudaMemcpyToSymbol(g_axis_tma_timeout, &z, sizeof(int));
  }
  return h;
}

}  // namespace tg
