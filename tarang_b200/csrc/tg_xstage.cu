// x-forward of a stage's products, the stage itself and the x-inverse of the next stage's fields in one
// kernel.
//
// Every one of the three works on whole columns (ky, kz): the passes transform them along x and the stage
// is pointwise, so the product spectra and the stage fields need not go through memory between them.  A
// block takes a few columns of all products: one group of threads per product loads its tile by TMA,
// transforms it in place (the two-step FFT of k_axis_tma) and leaves the kept rows; then every thread
// takes modes (all products of a mode from shared memory, the master state and the accumulator from
// global) and puts the stage's fields where the first products were; then a group per field transforms
// back, in place, and stores the tile by TMA.
//
// Bound: memory, and the serial phases of a block.  Per mode and stage the separate passes moved the
// products twice (written, read), the stage fields twice, and the rest as here; in FP64 at 256^3 (fluid)
// 1.18 GB a stage against 0.85.  Tiles of 64-byte rows (4 columns in FP64, 8 in FP32) leave shared memory
// and registers for 640 threads an SM.  At small grids it is three launches of a latency chain in one.
// Measured (B200): 226 us a stage at 256^3 FP64 against 87 + 106 + 61; the steps' times stand at
// xstage_fits.  Prefetching the state's rows into L2 while the products transform: FP64 fluid 64 x 256 x 256
// 68.6 us a stage without, 60.6 with it; 256^3 227 and 224.
#include <algorithm>
#include <cstring>

#include "tg_dft.cuh"
#include "tg_rk.cuh"
#include "tg_tma.cuh"
#include "tg_xstage.h"

namespace tg {

namespace {

// columns of a tile: 64-byte rows
template <typename R>
struct XW {
  static constexpr int v = 64 / (int)sizeof(cx<R>);
};
constexpr int kXPolls = 1 << 20;

struct XMaps {
  CUtensorMap src[8];
  CUtensorMap dst[6];
};

template <int PHYS>
struct XProd {
  static constexpr int v = PHYS == PH_FLUID ? 5 : 8;
};
// threads of a product's group
template <typename R, int R1>
struct XGroup {
  static constexpr int v = XW<R>::v * R1;
};
// resident blocks an SM the kernel is built for: 640 threads, 96 to 102 registers each
constexpr int x_occ(int threads) { return threads >= 640 ? 1 : 640 / threads; }

template <int G>
__device__ __forceinline__ void group_sync(int g) {
  if constexpr (G <= 32) {
    __syncwarp();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(G) : "memory");
  }
}

// row of the exchange: entry (k1, m) of the two-step FFT.  m is rotated by k1 so that the threads k1, k1 + 1,
// .. that read one m touch distinct banks (a row is 64 or 32 bytes)
template <typename R, int R2>
__device__ __forceinline__ int x_row(int k1, int m) {
  constexpr int SW = 1;  // two rows of 64 bytes a cycle of banks
  return k1 * R2 + (m ^ (k1 & SW));
}

template <typename R, int PHYS, int R1, int R2, int STAGE>
__global__ void __launch_bounds__(XProd<PHYS>::v * XGroup<R, R1>::v, x_occ(XProd<PHYS>::v * XGroup<R, R1>::v))
    k_xstage(RKArgs a, const __grid_constant__ XMaps tm, const cx<double>* __restrict__ twg, int us_all, int* wait_flag,
             int wait_short) {
  constexpr int L = R1 * R2, W = XW<R>::v, NP = XProd<PHYS>::v, NS = NState<PHYS>::v, G = XGroup<R, R1>::v;
  constexpr int CE = (int)sizeof(cx<R>) / 8;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((128u - (smem_u32(smem_raw) & 127u)) & 127u);
  uint64_t* bar = reinterpret_cast<uint64_t*>(base);           // [NP]
  int* fail = reinterpret_cast<int*>(base + 8 * NP);
  cx<R>* tw = reinterpret_cast<cx<R>*>(base + 128);             // e^{-2 pi i m / L}
  cx<R>* tiles = reinterpret_cast<cx<R>*>(base + 128 + ((L * sizeof(cx<R>) + 127) & ~(size_t)127));
  const Geo& geo = a.g;
  const int tid = threadIdx.x, g = tid / G, t = tid - g * G;
  const int slot = blockIdx.y, col0 = blockIdx.x * W;
  cx<R>* tile = tiles + (size_t)g * L * W;
  if (tid == 0) {
    for (int q = 0; q < NP; ++q) mbar_init(&bar[q], 1);
    *fail = 0;
    mbar_init_fence();
  }
  __syncthreads();
  pdl_wait();
  if (t == 0) {
    mbar_arrive_expect_tx(&bar[g], (unsigned)(L * W * sizeof(cx<R>)));
    tma_load_3d(tile, &tm.src[g], col0 * CE, 0, slot, &bar[g]);
  }
  {
    // the stage's rows of U0 and TOT (64 bytes each) on their way to L2 while the products transform
    const long long gb = (long long)slot * geo.S + col0, gr = (long long)geo.nky * geo.kzp;
    constexpr int NF = (STAGE == 2 || STAGE == 3) ? 2 * NS : NS;
    for (int i = tid; i < geo.nkx * NF; i += NP * G) {
      const int c = i / geo.nkx, r1 = i - c * geo.nkx;
      const cx<double>* p = (c < NS ? a.U0[c] : a.TOT[c - NS]) + gb + r1 * gr;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
      if constexpr (W == 8) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 4));
    }
  }
  for (int i = tid; i < L; i += NP * G) tw[i] = cvt<R>(twg[i]);
  if (t == 0 && !mbar_wait_bounded(&bar[g], 0, wait_short ? 0 : kXPolls)) {
    *fail = 1;
    if (wait_flag) atomicExch(wait_flag, 1);
    mbar_wait_bounded(&bar[g], 0, kXPolls);  // let a late copy land before the block leaves
  }
  __syncthreads();  // twiddles; every tile is in, or the block leaves
  if (*fail) return;
  mbar_wait_bounded(&bar[g], 0, 64);  // the phase has completed: acquire the copied tile

  const int w = t % W, n = t / W;  // n: n2 of the first step, k1 of the second
  // ---- forward
  {
    cx<R> v[R1];
    if (n < R2) {
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) v[n1] = tile[(R2 * n1 + n) * W + w];
      DFT<R1, -1, R>::run(v);
    }
    group_sync<G>(g);
    if (n < R2) {
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) tile[x_row<R, R2>(k1, n) * W + w] = v[k1] * tw[(n * k1) & (L - 1)];
    }
    group_sync<G>(g);
    cx<R> u[R2];
#pragma unroll
    for (int m = 0; m < R2; ++m) u[m] = tile[x_row<R, R2>(n, m) * W + w];
    DFT<R2, -1, R>::run(u);
    group_sync<G>(g);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) {
      const int r = amap_row(geo.ax, n + R1 * k2);
      if (r >= 0) tile[r * W + w] = u[k2];
    }
  }
  __syncthreads();

  // ---- the stage, one mode a turn
  {
    const double dt = a.dt[(long long)slot * 8];
    double nus[NS], nuh[NS];
#pragma unroll
    for (int c = 0; c < NS; ++c) {
      nus[c] = a.nu_tab ? a.nu_tab[slot * 6 + c] : a.nu[c];
      nuh[c] = a.nuh[c];
    }
    const int r2 = col0 / geo.kzp, l30 = col0 - r2 * geo.kzp;  // the tile lies in one ky row (kzp % 8 == 0)
    const int kyi = geo_ky(geo, r2);
    const double ky = kyi * geo.kf1;
    const long long gb = (long long)slot * geo.S + col0, gr = (long long)geo.nky * geo.kzp;
    for (int i = tid; i < geo.nkx * W; i += NP * G) {
      const int r1 = i / W, ww = i - r1 * W, l3 = l30 + ww;
      const long long gi = gb + r1 * gr + ww;
      if (l3 >= geo.nkz) {
#pragma unroll
        for (int c = 0; c < NS; ++c) tiles[(size_t)c * L * W + i] = mkc<R>(0, 0);
        continue;
      }
      cx<double> u0[NS], tot[NS];
#pragma unroll
      for (int c = 0; c < NS; ++c) u0[c] = a.U0[c][gi];
      if constexpr (STAGE == 2 || STAGE == 3) {
#pragma unroll
        for (int c = 0; c < NS; ++c) tot[c] = a.TOT[c][gi];
      }
      const int kxi = geo_kx(geo, r1);
      const double kx = kxi * geo.kf0, kz = l3 * geo.kf2;
      const double K2 = mode_k2(kx, ky, kz);
      cx<double> p[9], r[NS];
      p[2] = mkc<double>(0, 0);
#pragma unroll
      for (int q = 0; q < NP; ++q) p[q < 2 ? q : q + 1] = cvt<double>(tiles[(size_t)q * L * W + i]);
      const XDer dx{kx, 0};
      assemble<PHYS>(p, dx, ky, kz, r);
      sub_forces<PHYS>(a, gi, kxi, kyi, l3, kx, ky, kz, K2, r);
      project_rhs(r, NS, dx, ky, kz, K2);
      const bool keep = us_all || (a.FB != nullptr && kxi >= -a.fx && kxi <= a.fx && kyi >= -a.fy && kyi <= a.fy && l3 <= a.fz);
      double eh = 0, e1 = 0;
      cx<R> us[NS];
#pragma unroll
      for (int c = 0; c < NS; ++c) {
        if (c == 0 || nus[c] != nus[c - 1] || nuh[c] != nuh[c - 1]) {
          const double nuk = mode_nu(nus[c], nuh[c], K2);
          eh = exp(-nuk * 0.5 * dt * K2);
          if constexpr (STAGE == 1) e1 = exp(-nuk * dt * K2);
        }
        const cx<R> u = cvt<R>(stage_field<STAGE>(u0[c], r[c], dt, eh));
        if constexpr (STAGE != 7) a.TOT[c][gi] = stage_total<STAGE>(STAGE == 1 ? mkc<double>(0, 0) : tot[c], r[c], dt, eh, e1);
        us[c] = u;
        if (keep) reinterpret_cast<cx<R>*>(a.US[c])[gi] = u;
      }
      // the fields of the x-inverse: z+ = U + B and z- = U - B for MHD
#pragma unroll
      for (int c = 0; c < NS; ++c) {
        cx<R> x = us[c];
        if constexpr (PHYS == PH_MHD) x = c < 3 ? us[c] + us[3 + c] : us[c - 3] - us[c];
        tiles[(size_t)c * L * W + i] = x;
      }
    }
  }
  __syncthreads();

  // ---- inverse of the stage's fields
  if (g >= NS) return;
  {
    cx<R> v[R1];
    if (n < R2) {
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1) {
        const int r = amap_row(geo.ax, R2 * n1 + n);
        v[n1] = r >= 0 ? tile[r * W + w] : mkc<R>(0, 0);
      }
      DFT<R1, +1, R>::run(v);
    }
    group_sync<G>(g);
    if (n < R2) {
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) tile[x_row<R, R2>(k1, n) * W + w] = v[k1] * conjc(tw[(n * k1) & (L - 1)]);
    }
    group_sync<G>(g);
    cx<R> u[R2];
#pragma unroll
    for (int m = 0; m < R2; ++m) u[m] = tile[x_row<R, R2>(n, m) * W + w];
    DFT<R2, +1, R>::run(u);
    group_sync<G>(g);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) tile[(n + R1 * k2) * W + w] = u[k2];
    fence_proxy_async_smem();
    group_sync<G>(g);
    if (t == 0) {
      tma_store_3d(&tm.dst[g], col0 * CE, 0, slot, tile);
      bulk_commit_group();
      bulk_wait_group_read0();
    }
  }
}

size_t xstage_smem(int L, size_t csz, int np) {
  return 128 + 128 + ((L * csz + 127) & ~(size_t)127) + (size_t)np * L * 64;
}

template <typename R, int PHYS, int R1, int R2>
cudaError_t run_xstage(const XStageLaunch& l, cudaStream_t s, bool* used) {
  constexpr int L = R1 * R2, NP = XProd<PHYS>::v, NS = NState<PHYS>::v, CE = (int)sizeof(cx<R>) / 8, W = XW<R>::v;
  const Geo& g = l.rk.g;
  const unsigned long long ncols = (unsigned long long)g.nky * g.kzp;
  const int nact = l.rk.nact > 0 ? l.rk.nact : 1;
  XMaps tm;
  std::memset(&tm, 0, sizeof(tm));
  for (int q = 0; q < NP + NS; ++q) {
    const void* p = q < NP ? l.src[q] : l.dst[q - NP];
    if (!tma_map_3d(q < NP ? &tm.src[q] : &tm.dst[q - NP], p, ncols * CE, L, nact, ncols * sizeof(cx<R>),
                    ncols * L * sizeof(cx<R>), W * CE, L))
      return cudaSuccess;
  }
  const size_t smem = xstage_smem(L, sizeof(cx<R>), NP);
  auto go = [&](auto kern) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    if (e != cudaSuccess) return e;
    return launch_pdl(kern, dim3((unsigned)(ncols / W), nact), NP * XGroup<R, R1>::v, smem, s, l.rk, tm, l.tw, l.us_all,
                      l.wait_flag, l.wait_short);
  };
  *used = true;
  switch (l.rk.stage) {
    case 1: return go(k_xstage<R, PHYS, R1, R2, 1>);
    case 2: return go(k_xstage<R, PHYS, R1, R2, 2>);
    case 3: return go(k_xstage<R, PHYS, R1, R2, 3>);
    case 7: return go(k_xstage<R, PHYS, R1, R2, 7>);
    default: *used = false; return cudaSuccess;
  }
}

template <typename R, int PHYS>
cudaError_t run_xstage_l(const XStageLaunch& l, cudaStream_t s, bool* used) {
  switch (l.rk.g.N1) {
    case 32: return run_xstage<R, PHYS, 8, 4>(l, s, used);
    case 64: return run_xstage<R, PHYS, 8, 8>(l, s, used);
    case 128:
      if constexpr (sizeof(R) == 8 && PHYS == PH_FLUID) return run_xstage<R, PHYS, 16, 8>(l, s, used);
      return cudaSuccess;
    case 256:
      if constexpr (sizeof(R) == 8 && PHYS == PH_FLUID) return run_xstage<R, PHYS, 16, 16>(l, s, used);
      return cudaSuccess;
    default: return cudaSuccess;
  }
}

template <typename R>
cudaError_t run_xstage_p(const XStageLaunch& l, cudaStream_t s, bool* used) {
  switch (l.phys) {
    case PH_FLUID: return run_xstage_l<R, PH_FLUID>(l, s, used);
    case PH_MHD: return run_xstage_l<R, PH_MHD>(l, s, used);
    case PH_SCALAR: return run_xstage_l<R, PH_SCALAR>(l, s, used);
    default: return cudaSuccess;
  }
}

}  // namespace

// The lines.  One request: a grid whose tiles fit one wave is a latency chain, where three launches in one win
// whatever the kernel's own rate: two blocks an SM, or one of the 512 threads of the FP32 MHD and scalar forms (64 x 96
// x 64, 186 tiles, fused / separate, us a step: 176.1 / 168.3 and 165.6 / 162.6; 64 x 64 x 128, 252 tiles, 149.8 / 142.5
// and 133.6 / 133.4).  A larger grid is taken where the fused kernel, at 20 warps an SM, still beats the three passes at
// 24 to 48: FP64 fluid with N1 = 256 or 64.  Steps measured (fused / separate, us, the y and z passes one by one): 32^3
// FP32 fluid 59.6 / 66.5, MHD 67.8 / 76.0; 64^3 FP64 fluid 94.5 / 102.0, scalar 124 / 135, FP32 MHD 98 / 107;
// 256 x 64 x 64 FP64 256 / 282; 256^3 FP64 2806 / 3000; 64 x 256 x 256 FP64 806 / 829; and against it 64 x 256 x 256
// FP32 500 / 475, MHD 901 / 846, 128^3 FP64 463 / 448, 256^3 FP32 1686 / 1647.
// A batch, where one request is taken: as long as its tiles stay within two waves (one of the 512-thread forms),
// and at any size for FP64 with N1 = 64.  Steps of 4 and of 16 requests: 32^3 FP64 fluid 98 / 109 and 199 / 188, 64^3
// FP32 fluid 181 / 186 and 546 / 524, 64^3 FP64 scalar 438 / 448 and 1507 / 1522; 32 x 32 x 128 FP32 MHD 229 / 207 and
// 657 / 563, scalar 202 / 177 and 569 / 472, FP64 MHD 281 / 277 and 884 / 817.
// Both ways give the same bits (tg_rk.cuh), so a result does not depend on the batch.
bool xstage_fits(const Geo& g, int phys, int prec, int nact) {
  if (!axis_tma_enabled() || g.basis != 0 || g.x0 != 0 || phys == PH_RB || g.kzp % 8 != 0) return false;
  const bool f64 = prec == F64, fluid = phys == PH_FLUID;
  const bool have = g.N1 == 32 || g.N1 == 64 || (f64 && fluid && (g.N1 == 128 || g.N1 == 256));
  if (!have) return false;
  const long long tiles = (long long)g.nky * g.kzp / (f64 ? XW<double>::v : XW<float>::v);
  if (f64 && fluid && (g.N1 == 64 || g.N1 == 256)) return true;
  const bool wide = !f64 && !fluid;  // 512 threads
  if (tiles > (wide ? 148 : 2 * 148)) return false;
  if (nact <= 1 || (f64 && g.N1 == 64)) return true;
  return tiles * nact <= (wide ? 148 : (f64 && fluid ? 2 * 4 * 148 : 2 * 2 * 148));
}

cudaError_t launch_xstage(const XStageLaunch& l, cudaStream_t s, bool* used) {
  *used = false;
  if (l.rk.nact > 65535) return cudaSuccess;
  return l.prec == F64 ? run_xstage_p<double>(l, s, used) : run_xstage_p<float>(l, s, used);
}

}  // namespace tg
