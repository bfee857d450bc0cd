// SCFT x-pass of the pipeline in FP32 (sine / cosine transforms along x, scft_tr.cc:440-639) as a
// folded matrix product in registers.  Folding as in k_axis_r2r_dmma (tg_fft_dmma.cuh): step j takes a
// pair of inputs (p, q) per column, the sum and the difference of the points j and N-1-j (forward) or
// the coefficients 2 j and 2 j + 1 (inverse), and adds c0[i] p to A_i and c1[i] q to B_i, i < RT;
// the rows are A and B (forward) or A + B and +-(A - B) (inverse).  Half the multiply-adds of the full
// matrix.
//
// A thread owns two complex columns and 2 RT accumulators a column; the coefficients of the row tile
// are broadcast from shared memory; the inputs are copied by cp.async into the thread's own
// shared-memory ring, kFoldAhead - 1 steps ahead (two warps a scheduler at these registers do not
// hide a load), so a block has no barrier in its loop.  re and im are multiplied by one packed
// instruction.  The limits are the FP32 pipe and shared memory into the registers (128 bytes a cycle and SM,
// a broadcast counts for every lane: 56 cycles a step and warp against 44 of the pipe at RT = 22); what
// bounds a launch is latency at those few warps: issue slots 41 % used at 129 x 256 x 256, 34 % at
// 65 x 128 x 128 forward, 17 % inverse (ncu).
// Measured (B200, CUDA events around a launch; in brackets the 3xTF32 tensor-core form): 129 x 256 x 256
// forward of nine fields 115 us [134], 65 x 128 x 128 16.6 [26.1], inverse of four 17.1 [19.4];
// 33 x 256 x 256 24.8 [47.7] and 19.5 [21.2].  Row groups of one block sharing one staged copy of the
// inputs, a barrier a stage: 127 us and 22.9.
#pragma once

#include "tg_fft.cuh"

namespace tg {

__device__ __forceinline__ cx<float> fma_rc(float t, cx<float> x, cx<float> a) {
#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ >= 1000)
  return c2(__ffma2_rn(make_float2(t, t), f2(x), f2(a)));
#else
  return mkc<float>(fmaf(t, x.x, a.x), fmaf(t, x.y, a.y));
#endif
}

constexpr int kFoldThreads = 128;
constexpr int kFoldCols = 2 * kFoldThreads;  // complex columns of a block, two a thread
constexpr int kFoldAhead = 8;                // steps in the ring

// Even column counts and strides and 16-byte aligned buffers (run_r2r_fold).
// grid (column blocks, nbatch, nfields * ntile)
template <typename Ri, int RT, bool FWD>
__global__ void __launch_bounds__(kFoldThreads, RT <= 11 ? 3 : 2)
    k_axis_r2r_fold(AxisArgs a, PtrSet ps, R2RArgs r, int N, int ntile) {
  pdl_wait();
  constexpr int D = kFoldAhead;
  constexpr int RP = (RT + 3) / 4 * 4, TP = 2 * RP;  // c0 and c1 of a step, each a whole number of 16 bytes
  constexpr int NQ = (int)sizeof(cx<Ri>) / 8;        // 16-byte pieces of a thread's two columns
  constexpr unsigned QB = kFoldThreads * 16, RB = NQ * QB;  // a row of the ring: [NQ][kFoldThreads] pieces
  extern __shared__ __align__(16) unsigned char smem_raw[];
  unsigned char* ring = smem_raw + (size_t)threadIdx.x * 16;  // [D][2] rows
  float* Ts = reinterpret_cast<float*>(smem_raw + (size_t)D * 2 * RB);  // [steps][TP]
  const int f = blockIdx.z / ntile, tile = blockIdx.z - f * ntile;
  const int kind = r.kind[f];
  const int sine = kind & 1;
  const int nrows = r.mat_rows[kind], nin = r.mat_cols[kind];
  const int H = (N + 1) / 2;
  const int steps = FWD ? H : (nin + 1) / 2;
  const int i0 = tile * RT;
  const int col = blockIdx.x * kFoldCols + 2 * threadIdx.x;
  const bool any = col < a.ncols;
  const cx<Ri>* src = reinterpret_cast<const cx<Ri>*>(ps.src[f]) + (long long)blockIdx.y * a.sb + col;
  const unsigned ring_s = (unsigned)__cvta_generic_to_shared(ring);
  auto copy = [&](unsigned off, const cx<Ri>* p) {
    if constexpr (NQ == 1) {
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring_s + off), "l"(p) : "memory");
    } else {
#pragma unroll
      for (int c = 0; c < 2; ++c)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ring_s + off + QB * c), "l"(p + c) : "memory");
    }
  };
  auto column = [&](const unsigned char* row, int c) {
    return reinterpret_cast<const cx<Ri>*>(row + (NQ == 2 ? QB * c : 8 * c));
  };
  // step j's input rows: forward the points j and N - 1 - j, inverse the coefficients 2 j and 2 j + 1;
  // the second of an odd count's last step is zero
  const int pairs = (FWD ? N : nin) / 2;
  const cx<Ri>* pu = src;
  const cx<Ri>* pv = src + (FWD ? (N - 1) * a.sr : a.sr);
  unsigned wr = 0, rd = 0;  // ring offsets of the step to copy and of the step to read
  int jc = 0;
  auto copy_step = [&]() {
    if (any && jc < steps) {
      copy(wr, pu);
      if (jc < pairs) {
        copy(wr + RB, pv);
      } else {
#pragma unroll
        for (int c = 0; c < 2; ++c) *const_cast<cx<Ri>*>(column(ring + wr + RB, c)) = mkc<Ri>(0, 0);
      }
      pu += FWD ? a.sr : 2 * a.sr;
      pv += FWD ? -a.sr : 2 * a.sr;
    }
    ++jc;
    wr = wr == (D - 1) * 2 * RB ? 0 : wr + 2 * RB;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int j = 0; j < D - 1; ++j) copy_step();
  // c0 goes with the sum (forward) or the even coefficients (inverse), c1 with the difference or the
  // odd ones; a sine's even rows take the difference, and the middle point of an odd N has none
  const double* M = r.mat[kind];
#pragma unroll 4
  for (int e = threadIdx.x; e < steps * TP; e += kFoldThreads) {
    const int j = e / TP, m = e - j * TP, h = m >= RP, ii = m - h * RP, i = i0 + ii;
    const int k = FWD ? j : 2 * j + h, row = FWD ? 2 * i + (h ^ sine) : i;
    const bool mid = FWD && h && 2 * j == N - 1;
    Ts[e] = (ii < RT && k < nin && row < (FWD ? nrows : H) && !mid) ? (float)M[(size_t)k * nrows + row] : 0.0f;
  }
  __syncthreads();
  if (!any) return;
  cx<float> A[RT][2], B[RT][2];
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int c = 0; c < 2; ++c) A[i][c] = B[i][c] = mkc<float>(0, 0);
  const float4* t = reinterpret_cast<const float4*>(Ts);
  for (int j = 0; j < steps; ++j, t += TP / 4) {
    copy_step();
    asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
    const unsigned char* s = ring + rd;
    rd = rd == (D - 1) * 2 * RB ? 0 : rd + 2 * RB;
    cx<float> p[2], q[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const cx<float> x = cvt<float>(*column(s, c)), y = cvt<float>(*column(s + RB, c));
      p[c] = FWD ? x + y : x;
      q[c] = FWD ? x - y : y;
    }
#pragma unroll
    for (int v = 0; v < RP / 4; ++v) {
      const float4 w = t[v];
      const float co[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (4 * v + i < RT)
#pragma unroll
          for (int c = 0; c < 2; ++c) A[4 * v + i][c] = fma_rc(co[i], p[c], A[4 * v + i][c]);
    }
#pragma unroll
    for (int v = 0; v < RP / 4; ++v) {
      const float4 w = t[RP / 4 + v];
      const float co[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (4 * v + i < RT)
#pragma unroll
          for (int c = 0; c < 2; ++c) B[4 * v + i][c] = fma_rc(co[i], q[c], B[4 * v + i][c]);
    }
  }
  cx<float>* dst = reinterpret_cast<cx<float>*>(ps.dst[f]) + (long long)blockIdx.y * a.db + col;
  const float sc = (float)a.scale;
  auto store = [&](int row, cx<float> w0, cx<float> w1) {
    cx<float>* p = dst + (long long)row * a.dr;
    *reinterpret_cast<float4*>(p) = make_float4(sc * w0.x, sc * w0.y, sc * w1.x, sc * w1.y);
  };
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    if (FWD) {
      const int ra = 2 * (i0 + i) + sine, rb = 2 * (i0 + i) + 1 - sine;
      if (ra < nrows) store(ra, A[i][0], A[i][1]);
      if (rb < nrows) store(rb, B[i][0], B[i][1]);
    } else {
      const int k = i0 + i;
      if (k < H) {
        store(k, A[i][0] + B[i][0], A[i][1] + B[i][1]);
        if (N - 1 - k != k) {
          if (sine) store(N - 1 - k, B[i][0] - A[i][0], B[i][1] - A[i][1]);
          else store(N - 1 - k, A[i][0] - B[i][0], A[i][1] - B[i][1]);
        }
      }
    }
  }
}

}  // namespace tg
