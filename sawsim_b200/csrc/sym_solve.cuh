// Triangular solves of the symmetric path (sym_front.cuh), one CTA per (front,
// frequency).  A' is symmetric, so the adjoint system is solved by the same two kernels.
//
// A front's pivots come in blocks with an interchange of their own (piv: the block's row
// each pivot came from) and inverted 16 x 16 diagonal sub-blocks, so a block is four
// short products at most instead of a 64-step substitution; it is staged in shared memory
// by one coalesced pass.  The rows outside the block take eight lanes each: 128 (complex64:
// 64) contiguous bytes per load.  Fronts of one block (the lower levels of the tree) also
// do their update rows here; the wider ones leave them to front_fwd_l21_kernel and
// front_bwd_u12_kernel, which spread them over more CTAs.
//   Bound by the latency of the loads in flight: with each lane's entries loaded as one
// batch before any is used, 5.5 ms for both sweeps of the 32x128 ME1 cell at 51 points;
// the compiler keeps one load in flight in a loop of unknown length (8.0 ms).
#pragma once

namespace ss {

// sum of acc over groups of eight lanes (the result in each of them)
template <class T>
__device__ __forceinline__ cplx<T> sum8(cplx<T> acc) {
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
  }
  return acc;
}

// this lane's part of a row's product with y (shared memory), eight elements in flight
template <class T>
__device__ __forceinline__ cplx<T> warp_dot(const cplx<T> *row, const cplx<T> *y, int n, int lane) {
  constexpr int U = 8;
  cplx<T> acc{0, 0};
  for (int t0 = lane; t0 < n; t0 += 32 * U) {
    cplx<T> v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = t0 + 32 * u < n ? ld_el(row + t0 + 32 * u) : cplx<T>{0, 0};
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (t0 + 32 * u < n) acc = acc + cmul(v[u], y[t0 + 32 * u]);
  }
  return acc;
}

// rows [r0, r1) with eight lanes each: use(r, sum of F[r][c0 + t] y[t], t < n), n <= 8 E.
// A lane's E entries of two rows (E > 4: of one) are loaded before any is used.  Every lane
// of a warp makes the same number of rounds.
template <int E, class T, class Use>
__device__ __forceinline__ void rows8_e(const cplx<T> *F, int ld, int r0, int r1, int c0, int n, const cplx<T> *y, Use use) {
  constexpr int R = E > 4 ? 1 : 2;
  const int grp = threadIdx.x >> 3, sub = threadIdx.x & 7, ng = blockDim.x >> 3;
  const int first = (threadIdx.x & ~31) >> 3;      // the warp's first group
  for (int rb = r0; rb + first < r1; rb += R * ng) {
    cplx<T> v[R][E];
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = rb + grp + i * ng;
      const cplx<T> *row = F + (int64_t)r * ld + c0;
#pragma unroll
      for (int e = 0; e < E; ++e) v[i][e] = r < r1 && sub + 8 * e < n ? ld_el(row + sub + 8 * e) : cplx<T>{0, 0};
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int r = rb + grp + i * ng;
      cplx<T> acc{0, 0};
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (sub + 8 * e < n) acc = acc + cmul(v[i][e], y[sub + 8 * e]);
      acc = sum8(acc);
      if (r < r1 && sub == 0) use(r, acc);
    }
  }
}
template <class T, class Use>
__device__ __forceinline__ void rows8(const cplx<T> *F, int ld, int r0, int r1, int c0, int n, const cplx<T> *y, Use use) {
  if (n <= 16)
    rows8_e<2, T>(F, ld, r0, r1, c0, n, y, use);
  else if (n <= 40)
    rows8_e<5, T>(F, ld, r0, r1, c0, n, y, use);
  else
    rows8_e<8, T>(F, ld, r0, r1, c0, n, y, use);
}

// the block's n x n entries at F into D (row stride n + 1), eight lanes per row
template <class T>
__device__ __forceinline__ void stage_block(cplx<T> *D, const cplx<T> *F, int ld, int n) {
  const int grp = threadIdx.x >> 3, sub = threadIdx.x & 7, ng = blockDim.x >> 3;
  for (int r = grp; r < n; r += ng) {
    cplx<T> v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) v[e] = sub + 8 * e < n ? ld_el(F + (int64_t)r * ld + sub + 8 * e) : cplx<T>{0, 0};
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (sub + 8 * e < n) D[r * (n + 1) + sub + 8 * e] = v[e];
  }
}

// v (n entries, shared memory) <- L^-1 v (LOWER) or U^-1 v of the staged block; ends with
// a barrier
template <class T, bool LOWER>
__device__ __forceinline__ void block_solve(const cplx<T> *D, cplx<T> *v, int n) {
  const int grp = threadIdx.x >> 3, sub = threadIdx.x & 7, ds = n + 1;
  const int nh = (n + kDiagB - 1) / kDiagB;
  for (int q = 0; q < nh; ++q) {
    const int h0 = kDiagB * (LOWER ? q : nh - 1 - q), hw = min(kDiagB, n - h0);
    // the inverted diagonal sub-block: 16 groups of eight lanes
    cplx<T> y{0, 0};
    if (threadIdx.x < 8 * kDiagB) {
      if (grp < hw) {
        const cplx<T> *row = D + (h0 + grp) * ds + h0;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int t = sub + 8 * e;
          if (LOWER ? t < grp : (t >= grp && t < hw)) y = y + cmul(row[t], v[h0 + t]);
        }
        if (LOWER && sub == 0) y = y + v[h0 + grp];
      }
      y = sum8(y);
    }
    __syncthreads();
    if (threadIdx.x < 8 * kDiagB && grp < hw && sub == 0) v[h0 + grp] = y;
    __syncthreads();
    // the block's other rows
    const int r0 = LOWER ? h0 + hw : 0, r1 = LOWER ? n : h0;
    if (r1 > r0) {
      rows8_e<2, T>(D, ds, r0, r1, h0, hw, v + h0, [&](int r, cplx<T> s) { v[r] = v[r] - s; });
      __syncthreads();
    }
  }
}

// Forward: v = b[pivots] + the children's update vectors, L11 y = P v block by block;
// the update rows receive v - L21 y (one block) or v (more).  y overwrites x[pivots].
template <class T>
__global__ void __launch_bounds__(256) sym_fwd_kernel(FrontArgs<T> a, const cd *__restrict__ b, cd *__restrict__ x,
                                                      cplx<T> *__restrict__ wv, int64_t wstride, int maxb) {
  if (a.active && !a.active[blockIdx.y]) return;   // converged in the Krylov loop
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T> *D = reinterpret_cast<cplx<T> *>(smem_raw);
  cplx<T> *v = D + maxb * (maxb + 1);
  const int f = a.fronts[blockIdx.x], fq = blockIdx.y;
  const int k = a.k[f], m = a.m[f], ld = a.ld[f];
  const cplx<T> *F = a.arena + (int64_t)fq * a.stride + a.off[f];
  const int64_t p0 = a.p0[f];
  const int *piv = a.piv + (int64_t)fq * a.n + p0;
  const int bs = sym_block(k);
  int pv = threadIdx.x < min(bs, k) ? piv[threadIdx.x] : 0;      // the block's interchange, one block ahead
  stage_block<T>(D, F, ld, min(bs, k));
  for (int i = threadIdx.x; i < m; i += blockDim.x)
    v[i] = i < k ? to_t<T>(b[(int64_t)fq * a.n + p0 + i]) : cplx<T>{0, 0};
  cplx<T> *w = wv + (int64_t)fq * wstride;
  for (int64_t cc = a.child_ptr[f]; cc < a.child_ptr[f + 1]; ++cc) {
    const int ch = a.child[cc];
    const int nn = a.m[ch] - a.k[ch];
    const int *rel = a.relpos + a.relpos_ptr[ch];
    const cplx<T> *wc = w + a.relpos_ptr[ch];
    __syncthreads();
    for (int i = threadIdx.x; i < nn; i += blockDim.x) v[rel[i]] = v[rel[i]] + wc[i];
  }
  w += a.relpos_ptr[f] - k;
  for (int b0 = 0; b0 < k; b0 += bs) {
    const int n = min(bs, k - b0);
    if (b0) stage_block<T>(D, F + (int64_t)b0 * (ld + 1), ld, n);
    __syncthreads();
    cplx<T> g{0, 0};
    if (threadIdx.x < n) g = v[b0 + pv];
    if (b0 + bs + (int)threadIdx.x < min(k, b0 + 2 * bs)) pv = piv[b0 + bs + threadIdx.x];
    __syncthreads();
    if (threadIdx.x < n) v[b0 + threadIdx.x] = g;
    __syncthreads();
    block_solve<T, true>(D, v + b0, n);
    if (k <= kNarrowK) {
      rows8<T>(F, ld, k, m, 0, n, v, [&](int r, cplx<T> s) { w[r] = v[r] - s; });
    } else {
      rows8<T>(F, ld, b0 + n, k, b0, n, v + b0, [&](int r, cplx<T> s) { v[r] = v[r] - s; });
      __syncthreads();
    }
  }
  if (k > kNarrowK)
    for (int r = k + threadIdx.x; r < m; r += blockDim.x) w[r] = v[r];
  for (int i = threadIdx.x; i < k; i += blockDim.x) x[(int64_t)fq * a.n + p0 + i] = cd{(double)v[i].x, (double)v[i].y};
}

// Backward (levels run root first): U11 z = y - U12 x_U, the last block first; the U12
// product is done here for fronts of one block.  z overwrites x[pivots].
template <class T>
__global__ void __launch_bounds__(256) sym_bwd_kernel(FrontArgs<T> a, cd *__restrict__ x, int maxb) {
  if (a.active && !a.active[blockIdx.y]) return;   // converged in the Krylov loop
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cplx<T> *D = reinterpret_cast<cplx<T> *>(smem_raw);
  cplx<T> *z = D + maxb * (maxb + 1);
  const int f = a.fronts[blockIdx.x], fq = blockIdx.y;
  const int k = a.k[f], m = a.m[f], ld = a.ld[f];
  const cplx<T> *F = a.arena + (int64_t)fq * a.stride + a.off[f];
  const int64_t p0 = a.p0[f];
  cd *xf = x + (int64_t)fq * a.n;
  const int bs = sym_block(k), last = (k - 1) / bs * bs;
  stage_block<T>(D, F + (int64_t)last * (ld + 1), ld, k - last);
  for (int i = threadIdx.x; i < k; i += blockDim.x) z[i] = to_t<T>(xf[p0 + i]);
  if (k <= kNarrowK && m > k) {
    cplx<T> *xu = z + k;
    const int64_t *rows = a.rows + a.rows_ptr[f] + k;
    for (int i = threadIdx.x; i < m - k; i += blockDim.x) xu[i] = to_t<T>(xf[rows[i]]);
    __syncthreads();
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int r = threadIdx.x >> 5; r < k; r += nw) {
      cplx<T> acc = warp_dot(F + (int64_t)r * ld + k, xu, m - k, lane);
      for (int o = 16; o > 0; o >>= 1) {
        acc.x += __shfl_down_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_down_sync(0xffffffffu, acc.y, o);
      }
      if (lane == 0) z[r] = z[r] - acc;
    }
  }
  for (int b0 = last; b0 >= 0; b0 -= bs) {
    const int n = min(bs, k - b0);
    if (b0 != last) stage_block<T>(D, F + (int64_t)b0 * (ld + 1), ld, n);
    __syncthreads();
    block_solve<T, false>(D, z + b0, n);
    rows8<T>(F, ld, 0, b0, b0, n, z + b0, [&](int r, cplx<T> s) { z[r] = z[r] - s; });
  }
  __syncthreads();
  for (int i = threadIdx.x; i < k; i += blockDim.x) xf[p0 + i] = cd{(double)z[i].x, (double)z[i].y};
}

}  // namespace ss
