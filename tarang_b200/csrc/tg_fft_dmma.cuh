// SCFT x-pass of the pipeline in FP64 (sine / cosine transforms along x, scft_tr.cc:440-639) as a
// folded matrix product on the FP64 matrix instructions (mma.sync m8n8k4 f64: exact FP64 fused
// multiply-adds; tcgen05 has no FP64 kind).
//
// Folding: cos(pi m (2n+1) / 2N) and sin(..) change only their sign, by the parity of m, under
// n -> N-1-n, so
//   forward (points to coefficients)  even and odd rows m need only s_n = x_n + x_(N-1-n) and
//       d_n = x_n - x_(N-1-n), n < H = ceil(N/2)  (cosine: even rows s, odd rows d; sine the
//       other way round), and
//   inverse (coefficients to points)  with E_k, O_k the sums over the even and the odd m, the points
//       k and N-1-k are E + O and +-(E - O),
// which halves the multiply-adds of the full matrix.  Both directions are one product per set
// h = 0, 1: C_h[i][col] = sum_j c_h[i][j] b_h[j][col] with (b_0, b_1) = (s, d) or the even and odd
// coefficients, over the real columns (re, im interleaved).
//
// Bound: the FP64 pipe.  A thread-per-column form (accumulators and broadcast coefficients in
// registers) is not: each multiply-add takes its coefficient from shared memory, whose 128 bytes a
// cycle and SM into the registers capped it at 45 % of the pipe; and plain fused multiply-adds reach
// 28.7 TFLOP/s where the matrix instruction reaches 36.6 (both measured, independent chains, B200).
// Here a warp holds all rows of 8 real columns (2 MT tiles of 8 x 8), so a fragment of b feeds MT
// instructions; 16 warps (four a scheduler) cover each other's barriers and stores.  Input rows arrive by cp.async in stages of 8 pairs, three stages
// ahead, without a break from one column tile to the next; the coefficients of the block's rows are
// laid out in fragment order once per block, and blocks are persistent (one per SM).
// Measured (B200, CUDA events around a launch; in brackets the register-tiled product of the full
// matrix): 129 x 256 x 256 forward of nine fields 163 us [469] (23 TFLOP/s of folded work), inverse of
// four 89 [227]; 65 x 128 x 128 23.5 [42.1] and 18.2 [26.3].  What is left is the barrier of every
// stage and the stores, behind which the pipe idles.  Half the warps with twice the columns: 197, 101.
#pragma once

#include "tg_fft.cuh"

namespace tg {

constexpr int kDmThreads = 512;             // 16 warps of 8 real columns
constexpr int kDmCols = 64;                 // complex columns of a tile
constexpr int kDmPairs = 8;                 // pairs of input rows of a stage
constexpr int kDmStages = 4;
constexpr int kDmPitch = 2 * kDmCols + 8;   // doubles of a staged row: rows 64 bytes apart mod 256
constexpr int kDmStageD = 2 * kDmPairs * kDmPitch;

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// grid (P, nbatch, nfields * nrb): block (x, b, f, rb) takes the column tiles x, x + P, .. of batch b,
// field f, and the row pairs [8 MT rb, 8 MT (rb + 1)).
template <int MT, bool FWD>
__global__ void __launch_bounds__(kDmThreads, 1) k_axis_r2r_dmma(AxisArgs a, PtrSet ps, R2RArgs r, int N, int nrb) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* ring = reinterpret_cast<double*>(smem_raw);  // [stage][u rows, v rows][pitch]
  double* Af = ring + kDmStages * kDmStageD;           // [k4][set][mt][32]
  const int f = blockIdx.z / nrb, rbk = blockIdx.z - f * nrb;
  const int kind = r.kind[f];
  const int sine = kind & 1;
  const int nrows = r.mat_rows[kind], nin = r.mat_cols[kind];
  const int H = (N + 1) / 2;
  const int npair = FWD ? H : (nin + 1) / 2;           // pairs of input rows
  const int nst = (npair + kDmPairs - 1) / kDmPairs;   // stages of a column tile
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gid = lane >> 2, tig = lane & 3;
  const int ntiles = (a.ncols + kDmCols - 1) / kDmCols, P = (int)gridDim.x;
  const int my_tiles = (ntiles - (int)blockIdx.x + P - 1) / P, total = my_tiles * nst;
  const cx<double>* src = reinterpret_cast<const cx<double>*>(ps.src[f]) + (long long)blockIdx.y * a.sb;
  cx<double>* dst = reinterpret_cast<cx<double>*>(ps.dst[f]) + (long long)blockIdx.y * a.db;

  // the copy cursor: this thread's pair (row qi of a stage's u rows and of its v rows) and complex
  // column, stage by stage and tile by tile; rows past the last pair, and the second row of an odd
  // count's last pair, are filled with zeros
  const int qi = tid >> 6, cc = tid & (kDmCols - 1);
  int ct = 0, cs = 0, cslot = 0, cj = qi, ccol = (int)blockIdx.x * kDmCols + cc;
  const long long rs = a.sr;
  const cx<double>* pu = src + (FWD ? (long long)qi * rs : 2LL * qi * rs) + ccol;
  const cx<double>* pv = src + (FWD ? (long long)(N - 1 - qi) * rs : (2LL * qi + 1) * rs) + ccol;
  const long long du = FWD ? kDmPairs * rs : 2LL * kDmPairs * rs, dv = FWD ? -kDmPairs * rs : 2LL * kDmPairs * rs;
  const unsigned dp0 = (unsigned)__cvta_generic_to_shared(ring + qi * kDmPitch + 2 * cc);
  auto copy_stage = [&]() {
    if (ct < my_tiles) {
      const bool lu = cj < npair && ccol < a.ncols, lv = lu && (FWD ? 2 * cj != N - 1 : 2 * cj + 1 < nin);
      const unsigned dp = dp0 + cslot * (unsigned)(kDmStageD * sizeof(double));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dp), "l"(lu ? pu : src), "r"(lu ? 16 : 0)
                   : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dp + (unsigned)(kDmPairs * kDmPitch * sizeof(double))),
                   "l"(lv ? pv : src), "r"(lv ? 16 : 0)
                   : "memory");
      cslot = cslot == kDmStages - 1 ? 0 : cslot + 1;
      if (++cs == nst) {
        cs = 0;
        ++ct;
        cj = qi;
        ccol += P * kDmCols;
        pu += P * kDmCols - (nst - 1) * du;
        pv += P * kDmCols - (nst - 1) * dv;
      } else {
        cj += kDmPairs;
        pu += du;
        pv += dv;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // coefficients in fragment order: A(row gid, k tig).  A sine's even rows take the difference; the
  // middle point of an odd N has none
  const double* M = r.mat[kind];
  const int nk4 = nst * (kDmPairs / 4);
#pragma unroll 4
  for (int e = tid; e < nk4 * 2 * MT * 32; e += kDmThreads) {
    const int ln = e & 31, mt = (e >> 5) % MT, hk = (e >> 5) / MT, h = hk & 1, k4 = hk >> 1;
    const int j = 4 * k4 + (ln & 3), i = 8 * (rbk * MT + mt) + (ln >> 2);
    const int k = FWD ? j : 2 * j + h, row = FWD ? 2 * i + (h ^ sine) : i;
    const bool mid = FWD && h && 2 * j == N - 1;
    Af[e] = (j < npair && k < nin && row < (FWD ? nrows : H) && !mid) ? M[(size_t)k * nrows + row] : 0.0;
  }

  pdl_wait();
#pragma unroll
  for (int it = 0; it < kDmStages - 1; ++it) copy_stage();
  double c[2][MT][2];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int m = 0; m < MT; ++m) c[h][m][0] = c[h][m][1] = 0.0;
  const double sc = a.scale;
  int ks = 0, tile = (int)blockIdx.x, slot = 0;
  const double* s0 = ring + tig * kDmPitch + warp * 8 + gid;
  auto k4_step = [&](const double* s, const double* A) {
    const double x = s[0], y = s[kDmPairs * kDmPitch];
    const double b[2] = {FWD ? x + y : x, FWD ? x - y : y};
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int m = 0; m < MT; ++m) dmma(c[h][m], A[(h * MT + m) * 32], b[h]);
  };
  for (int it = 0; it < total; ++it) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kDmStages - 2) : "memory");
    __syncthreads();  // stage `it` is in for every thread, and every warp is done with stage it - 1
    const double* s = s0 + slot * kDmStageD;
    slot = slot == kDmStages - 1 ? 0 : slot + 1;
    const double* A = Af + (size_t)(kDmPairs / 4 * ks) * 2 * MT * 32 + lane;
    k4_step(s, A);
    copy_stage();  // behind the first products, so that its address work overlaps them
#pragma unroll
    for (int k4 = 1; k4 < kDmPairs / 4; ++k4)
      if (kDmPairs * ks + 4 * k4 < npair) k4_step(s + 4 * k4 * kDmPitch, A + k4 * 2 * MT * 32);
    if (++ks == nst) {
      ks = 0;
      // lane (gid, tig): row gid, complex column tig
      const int col = tile * kDmCols + warp * 4 + tig;
      if (col < a.ncols) {
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          const int i = 8 * (rbk * MT + m) + gid;
          const cx<double> e = mkc<double>(c[0][m][0], c[0][m][1]), o = mkc<double>(c[1][m][0], c[1][m][1]);
          if (FWD) {
            const int ra = 2 * i + sine, rb = 2 * i + 1 - sine;
            if (ra < nrows) dst[(long long)ra * a.dr + col] = sc * e;
            if (rb < nrows) dst[(long long)rb * a.dr + col] = sc * o;
          } else if (i < H) {
            dst[(long long)i * a.dr + col] = sc * (e + o);
            if (N - 1 - i != i) dst[(long long)(N - 1 - i) * a.dr + col] = sc * (sine ? o - e : e - o);
          }
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) c[h][m][0] = c[h][m][1] = 0.0;
      tile += P;
    }
  }
}

}  // namespace tg
