// Fronts of a complex symmetric system.
//
// The condensed FEM systems are complex symmetric up to one positive factor per
// potential column (K_phiu = s K_uphi^T), so with the scaling of sym_scale.cuh
// A' = A'^T to rounding, and so is every update block F22.  On this path
//   * a front is eliminated in pivot blocks of at most kNarrowK rows, each a small front
//     of its own: F11 (the block) is factored with row interchanges inside the block,
//     L21 = F21 U11^-1 and U12 = L11^-1 P F12 are formed from F12 alone (F21 = F12^T),
//     and the rest of the front is updated right away;
//   * only the upper triangle of an update block F22 - L21 U12 is formed: half of the
//     general path's Schur operations and update-block traffic, and the pivot blocks of
//     a wide front cost half of its LU too;
//   * the first block of a front reads its children's update blocks (at most two)
//     through inverse row maps (front row -> child update row or -1) where it needs them:
//     F11 and F12 when they are assembled, F22 in the epilogue of the Schur update, so
//     F22 is written once and never zeroed, scattered into or copied.  The later blocks
//     read the front itself, in place, through the identity map: the same kernels.
// The maps are monotone, so upper entries come from upper entries.  A front's memory
// holds, for every pivot block, L and U of F11 in pivot order, U12 right of it and L21
// below it (its rows in front order): the row interchanges of a later block are not
// applied to the L21 rows of an earlier one, the solves apply each block's interchange
// when they reach it.
#pragma once

namespace ss {

// Upper triangle of F22 = (children) - L21 U12 in 64 x 64 tiles on the FP64 tensor
// cores: the K loop of front_dmma3_kernel<2, 2> (three real products per complex
// block); the children's entries are copied into the staged C tile by cp.async when
// the CTA starts (each entry from the one child that has it), so their latency
// overlaps the K loop; entries that both children have take the second one in the
// epilogue.  Tiles below the diagonal are not launched; a diagonal tile skips the
// entries below it.
constexpr int kSymCS = 65;
constexpr int sym_schur_smem() { return 64 * kSymCS * (int)sizeof(cd); }
__global__ void __launch_bounds__(128, 2) sym_schur_kernel(FrontArgs<double> a, const GemmTask *__restrict__ tasks) {
  constexpr int BS = 64 + 2;
  __shared__ __align__(16) cd As[2][64 * kDmmaAS];
  __shared__ __align__(16) cd Bs[2][kDmmaBK * BS];
  __shared__ int ir[2][64], ic[2][64];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *Cs = reinterpret_cast<cd *>(smem_raw);
  const GemmTask tk = tasks[blockIdx.x];
  const SymFront s = a.sf[tk.f];
  const int ld = s.ld;
  cd *arena = a.arena + (int64_t)blockIdx.y * a.stride;
  cd *F = arena + s.off;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int wm = wid >> 1, wn = wid & 1;
  const int g = lane >> 2, t = lane & 3;
  auto issue = [&](int buf, int kb) {
#pragma unroll
    for (int q = 0; q < 64 * kDmmaBK / 128; ++q) {
      const int idx = threadIdx.x + 128 * q;
      const int r = idx / kDmmaBK, k = idx % kDmmaBK;
      const int gr = tk.r0 + r, gk = kb + k;
      const bool ok = gr < tk.rhi && gk < tk.kk1;
      cp_async16_cd((uint32_t)__cvta_generic_to_shared(&As[buf][r * kDmmaAS + dmma_acol(r, k)]),
                    ok ? F + (int64_t)gr * ld + gk : F, ok ? 16u : 0u);
    }
#pragma unroll
    for (int q = 0; q < kDmmaBK * 64 / 128; ++q) {
      const int idx = threadIdx.x + 128 * q;
      const int k = idx / 64, c = idx % 64;
      const int gk = kb + k, gc = tk.c0 + c;
      const bool ok = gk < tk.kk1 && gc < tk.chi;
      cp_async16_cd((uint32_t)__cvta_generic_to_shared(&Bs[buf][k * BS + c]), ok ? F + (int64_t)gk * ld + gc : F,
                    ok ? 16u : 0u);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int nk = (tk.kk1 - tk.kk0 + kDmmaBK - 1) / kDmmaBK;
  if (s.nch) {
    sym_stage<double, 64, 64, 128, kSymCS>(Cs, s, arena, a.imap, tk, ir, ic);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  double p1[4][4][2], p2[4][4][2], p3[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) p1[i][j][e] = p2[i][j][e] = p3[i][j][e] = 0.0;
  issue(0, tk.kk0);
  for (int kc = 0; kc < nk; ++kc) {
    const int buf = kc & 1;
    if (kc + 1 < nk) {
      issue(buf ^ 1, tk.kk0 + (kc + 1) * kDmmaBK);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kDmmaBK; kk += 4) {
      cd av[4];
      double as[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int ar = wm * 32 + i * 8 + g;
        av[i] = As[buf][ar * kDmmaAS + dmma_acol(ar, kk + t)];
        as[i] = av[i].x + av[i].y;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const cd bv = Bs[buf][(kk + t) * BS + wn * 32 + j * 8 + g];
        const double bs = bv.x + bv.y;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          dmma(p1[i][j][0], p1[i][j][1], av[i].x, bv.x);
          dmma(p2[i][j][0], p2[i][j][1], av[i].y, bv.y);
          dmma(p3[i][j][0], p3[i][j][1], as[i], bs);
        }
      }
    }
    __syncthreads();
  }
  const bool two = s.nch > 1;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rl = wm * 32 + i * 8 + g, r = tk.r0 + rl;
    if (r >= tk.rhi) continue;
    cd *Fr = F + (int64_t)r * ld;
    const int i0 = s.nch ? ir[0][rl] : -1, i1 = two ? ir[1][rl] : -1;
    cd cv[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cl = wn * 32 + j * 8 + 2 * t + e, c = tk.c0 + cl;
        cv[j][e] = cd{0.0, 0.0};
        if (two && (i0 | i1) >= 0 && c >= r && c < tk.chi && (ic[0][cl] | ic[1][cl]) >= 0)
          cv[j][e] = ld_once(arena + s.cb[1] + (int64_t)i1 * s.cld[1] + ic[1][cl]);
      }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cl = wn * 32 + j * 8 + 2 * t + e, c = tk.c0 + cl;
        if (c < r || c >= tk.chi) continue;
        if (s.nch) cv[j][e] = Cs[rl * kSymCS + cl] + cv[j][e];
        const double re = p1[i][j][e] - p2[i][j][e];
        const double im = p3[i][j][e] - p1[i][j][e] - p2[i][j][e];
        st_el(Fr + c, cv[j][e] - cd{re, im});
      }
  }
}

// ------------------------------------------------------------------ pivot blocks
// A pivot block takes two kernels (and the Schur update) instead of the assembly, panel
// LU, row-swap, L21, U12 and panel-GEMM launches of every 32-pivot step:
//  * sym_pivot_kernel assembles F11 in shared memory, factors it and writes it in pivot
//    order;
//  * sym_panel_kernel takes one 64-column chunk of F12: it assembles the chunk in shared
//    memory, and one thread per column solves L11 y = P f (a column of U12) while
//    another takes the same f as a row of F21 = F12^T and solves z U11 = f^T (a row of
//    L21), 16 unknowns at a time in registers, the factors read as shared-memory
//    broadcasts.
// Row interchanges are implicit (a mask of eliminated rows); `piv` receives, for each
// pivot position, the front row it came from (the solve kernels gather).
constexpr int kPivotThreads = 128;
constexpr int kPanelColThreads = 128;
constexpr int kNarrowCS = 65;     // row stride of the chunk tile

// F11 of one pivot block with its arrowhead entries [a0, a1), or (c0 >= 0) the chunk of F12
// that starts at update column c0 with its entries
struct NarrowTask {
  int f, c0, a0, a1;
};
template <class T>
__host__ __device__ constexpr size_t pivot_smem(int k) {
  return ((size_t)k * (k + 1) + k) * sizeof(cplx<T>) + (size_t)3 * k * sizeof(int);
}
template <class T>
__host__ __device__ constexpr size_t panel_smem(int k) {
  return ((size_t)k * (k + 1) + (size_t)k * kNarrowCS + k) * sizeof(cplx<T>) + (size_t)k * sizeof(int);
}

// LU of the k x k matrix W (row stride ks, shared memory) with implicit row
// interchanges, one barrier per pivot: each warp owns the rows wid, wid + NW, ... and
// keeps the largest next-column entry of its open rows (four rows in flight).
// perm[j] = row of pivot j.  Returns the number of perturbed pivots.
template <class T, int NW>
__device__ __forceinline__ int narrow_lu(cplx<T> *W, int ks, int k, T tiny, int *perm) {
  __shared__ T s_v[2][NW];
  __shared__ int s_i[2][NW];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  {
    T best = (T)-1;
    int bi = 0;
    for (int r = wid + NW * lane; r < k; r += 32 * NW) {
      const T v = cabs1(W[r * ks]);
      if (v > best) best = v, bi = r;
    }
    for (int o = 16; o > 0; o >>= 1) {
      const T ov = __shfl_down_sync(0xffffffffu, best, o);
      const int oi = __shfl_down_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) best = ov, bi = oi;
    }
    if (lane == 0) s_v[1][wid] = best, s_i[1][wid] = bi;
    __syncthreads();
  }
  unsigned long long done = 0;
  bool pert_prev = false;
  int p_prev = 0, npert = 0;
  for (int j = 0; j < k; ++j) {
    const int par = (j & 1) ^ 1;
    T bv = s_v[par][0];
    int p = s_i[par][0];
#pragma unroll
    for (int q = 1; q < NW; ++q) {
      const T ov = s_v[par][q];
      const int oi = s_i[par][q];
      if (ov > bv || (ov == bv && oi < p)) bv = ov, p = oi;
    }
    if (p >= k || (done >> p & 1)) p = __ffsll((long long)~done) - 1;   // no comparable entry (NaN): any open row
    // the previous pivot's perturbed diagonal is read by no one any more
    if (pert_prev && tid == 0) W[p_prev * ks + j - 1] = cplx<T>{tiny, (T)0};
    const int c0 = j + 1 + lane, c1 = c0 + 32;
    cplx<T> pv = W[p * ks + j];
    const cplx<T> q0 = c0 < k ? W[p * ks + c0] : cplx<T>{0, 0}, q1 = c1 < k ? W[p * ks + c1] : cplx<T>{0, 0};
    const bool pert = cabs1(pv) < tiny;
    if (pert) pv = cplx<T>{tiny, (T)0};
    const cplx<T> inv = cdiv(cplx<T>{1, 0}, pv);
    if (tid == 0) perm[j] = p;
    npert += pert;
    pert_prev = pert;
    p_prev = p;
    done |= 1ull << p;
    T best = (T)-1;
    int bi = k;
    for (int rb = wid; rb < k; rb += 4 * NW) {
      cplx<T> l[4], v0[4], v1[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = min(rb + NW * i, k - 1);
        const cplx<T> *row = W + r * ks;
        l[i] = row[j];
        v0[i] = c0 < k ? row[c0] : cplx<T>{0, 0};
        v1[i] = c1 < k ? row[c1] : cplx<T>{0, 0};
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        l[i] = cmul(l[i], inv);
        v0[i] = cfms(v0[i], l[i], q0);
        v1[i] = cfms(v1[i], l[i], q1);
      }
      __syncwarp();      // every lane has read its row's multiplier
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = rb + NW * i;
        if (r >= k || (done >> r & 1)) continue;
        cplx<T> *row = W + r * ks;
        if (c0 < k) row[c0] = v0[i];
        if (c1 < k) row[c1] = v1[i];
        if (lane == 0) {
          row[j] = l[i];
          const T av = cabs1(v0[i]);
          if (av > best) best = av, bi = r;
        }
      }
    }
    if (lane == 0) s_v[j & 1][wid] = best, s_i[j & 1][wid] = bi;
    __syncthreads();
  }
  if (pert_prev && tid == 0) W[p_prev * ks + k - 1] = cplx<T>{tiny, (T)0};
  __syncthreads();
  return npert;
}

template <class T>
__global__ void __launch_bounds__(kPivotThreads)
    sym_pivot_kernel(FrontArgs<T> a, const NarrowTask *__restrict__ tasks, int nb, const uint16_t *__restrict__ apos,
                     const int *__restrict__ aslot) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NW = kPivotThreads / 32;
  const NarrowTask tk = tasks[blockIdx.x / nb];
  const int fq = blockIdx.x % nb;
  const SymFront &s = a.sf[tk.f];
  const int k = s.k, ks = k + 1;
  cplx<T> *W = reinterpret_cast<cplx<T> *>(smem_raw);
  int *perm = reinterpret_cast<int *>(W + k * ks + k), *ir = perm + k;
  cplx<T> *arena = a.arena + (int64_t)fq * a.stride;
  const double om = a.omega[fq];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nch = s.nch;
  if (nch) {
    for (int i = tid; i < k; i += kPivotThreads) {
      ir[i] = a.imap[s.imap[0] + i];
      ir[k + i] = nch > 1 ? a.imap[s.imap[1] + i] : -1;
    }
    __syncthreads();
    // the children's upper entries, mirrored
    for (int r = wid; r < k; r += NW)
      for (int c = r + lane; c < k; c += 32) {
        const cplx<T> v = sym_gather(s, arena, ir[r], ir[c], ir[k + r], ir[k + c]);
        W[r * ks + c] = v;
        W[c * ks + r] = v;
      }
  } else {
    for (int t = tid; t < k * ks; t += kPivotThreads) W[t] = cplx<T>{0, 0};
  }
  __syncthreads();
#pragma unroll 4
  for (int q = tk.a0 + tid; q < tk.a1; q += kPivotThreads) {
    const int r = apos[q] >> 6, c = apos[q] & 63;
    const cplx<T> v = W[r * ks + c] + to_t<T>(a_entry(a.Kc, a.Mc, a.Dc, aslot[q], om, a.beta));
    W[r * ks + c] = v;
    W[c * ks + r] = v;
  }
  __syncthreads();
  const int np = narrow_lu<T, NW>(W, ks, k, a.tiny, perm);
  if (np && tid == 0) atomicAdd(a.nperturb + fq, np);
  cplx<T> *F = arena + s.off;
  const int ld = s.ld;
  for (int r = wid; r < k; r += NW)
    for (int c = lane; c < k; c += 32) st_el(F + (int64_t)r * ld + c, W[perm[r] * ks + c]);
  for (int i = tid; i < k; i += kPivotThreads) a.piv[(int64_t)fq * a.n + s.p0 + i] = perm[i];
}

// H unknowns h0 .. h0 + hw of one triangular solve, v_i = (b_i - sum_{t < h0 + i} x_t
// C(t, i)) d_i.  LOWER: C = L[h0 + i][t], unit diagonal; else C = U[t][h0 + i] and d the
// reciprocal diagonal.  x points at the solved unknowns (stride xs).
template <class T, int H, bool LOWER>
__device__ __forceinline__ void narrow_block(cplx<T> (&v)[H], const cplx<T> *A, int ks, const cplx<T> *x, int64_t xs,
                                             int h0, int hw, const cplx<T> *dinv) {
#pragma unroll 4
  for (int t = 0; t < h0; ++t) {
    const cplx<T> xt = x[t * xs];
#pragma unroll
    for (int i = 0; i < H; ++i)
      if (i < hw) v[i] = cfms(v[i], LOWER ? A[(h0 + i) * ks + t] : A[t * ks + h0 + i], xt);
  }
#pragma unroll
  for (int i = 0; i < H; ++i) {
    if (i >= hw) break;
#pragma unroll
    for (int t = 0; t < i; ++t)
      v[i] = cfms(v[i], LOWER ? A[(h0 + i) * ks + h0 + t] : A[(h0 + t) * ks + h0 + i], v[t]);
    if (!LOWER) v[i] = cmul(v[i], dinv[h0 + i]);
  }
}
// one column of U12 in place at y (row stride ld, global memory)
template <class T, int H>
__device__ __forceinline__ void narrow_upper(const cplx<T> *A, int ks, cplx<T> *y, int64_t ld, int h0, int hw) {
  cplx<T> v[H];
#pragma unroll
  for (int i = 0; i < H; ++i) v[i] = i < hw ? ld_el(y + (h0 + i) * ld) : cplx<T>{0, 0};
  narrow_block<T, H, true>(v, A, ks, y, ld, h0, hw, nullptr);
#pragma unroll
  for (int i = 0; i < H; ++i)
    if (i < hw) st_el(y + (h0 + i) * ld, v[i]);
}
// one row of L21 in place in its column of the chunk tile
template <class T, int H>
__device__ __forceinline__ void narrow_lower(const cplx<T> *A, int ks, cplx<T> *z, const cplx<T> *dinv, int h0, int hw) {
  cplx<T> v[H];
#pragma unroll
  for (int i = 0; i < H; ++i) v[i] = i < hw ? z[(h0 + i) * kNarrowCS] : cplx<T>{0, 0};
  narrow_block<T, H, false>(v, A, ks, z, kNarrowCS, h0, hw, dinv);
#pragma unroll
  for (int i = 0; i < H; ++i)
    if (i < hw) z[(h0 + i) * kNarrowCS] = v[i];
}

template <class T>
__global__ void __launch_bounds__(kPanelColThreads, 3)
    sym_panel_kernel(FrontArgs<T> a, const NarrowTask *__restrict__ tasks, int nb, const uint16_t *__restrict__ apos,
                     const int *__restrict__ aslot) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NW = kPanelColThreads / 32;
  const NarrowTask tk = tasks[blockIdx.x / nb];
  const int fq = blockIdx.x % nb;
  const SymFront &s = a.sf[tk.f];
  const int k = s.k, ks = k + 1, nc = min(64, s.m - k - tk.c0);
  const int64_t ld = s.ld;
  cplx<T> *A = reinterpret_cast<cplx<T> *>(smem_raw);   // F11 in pivot order: L and U
  cplx<T> *ft = A + k * ks;                             // the chunk of F12, then of L21^T
  cplx<T> *dinv = ft + k * kNarrowCS;
  int *perm = reinterpret_cast<int *>(dinv + k);
  cplx<T> *arena = a.arena + (int64_t)fq * a.stride;
  cplx<T> *F = arena + s.off;
  const double om = a.omega[fq];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nch = s.nch;
  {
    const int64_t m0 = s.imap[0], m1 = s.imap[1];
    int j0[2], j1[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = lane + 32 * h;
      j0[h] = nch > 0 && c < nc ? a.imap[m0 + k + tk.c0 + c] : -1;
      j1[h] = nch > 1 && c < nc ? a.imap[m1 + k + tk.c0 + c] : -1;
    }
#pragma unroll 2
    for (int r = wid; r < k; r += NW) {
      const int i0 = nch > 0 ? a.imap[m0 + r] : -1, i1 = nch > 1 ? a.imap[m1 + r] : -1;
      const cplx<T> x0 = sym_gather(s, arena, i0, j0[0], i1, j1[0]), x1 = sym_gather(s, arena, i0, j0[1], i1, j1[1]);
      ft[r * kNarrowCS + lane] = x0;
      ft[r * kNarrowCS + lane + 32] = x1;
    }
    for (int r = wid; r < k; r += NW)
      for (int c = lane; c < k; c += 32) A[r * ks + c] = ld_el(F + r * ld + c);
    for (int i = tid; i < k; i += kPanelColThreads) perm[i] = a.piv[(int64_t)fq * a.n + s.p0 + i];
  }
  __syncthreads();
#pragma unroll 4
  for (int q = tk.a0 + tid; q < tk.a1; q += kPanelColThreads) {
    cplx<T> *d = ft + (apos[q] >> 6) * kNarrowCS + (apos[q] & 63);
    *d = *d + to_t<T>(a_entry(a.Kc, a.Mc, a.Dc, aslot[q], om, a.beta));
  }
  for (int i = tid; i < k; i += kPanelColThreads) dinv[i] = cdiv(cplx<T>{1, 0}, A[i * ks + i]);
  __syncthreads();
  // P F12 to the U12 rows (L21 is solved in place in the tile, U12 in global memory)
  cplx<T> *Y = F + k + tk.c0;
  for (int r = 16 + wid; r < k; r += NW)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = lane + 32 * h;
      if (c < nc) st_el(Y + r * ld + c, ft[perm[r] * kNarrowCS + c]);
    }
  const int c = tid & 63;
  cplx<T> first[16];      // the first unknowns' right-hand sides, read before L21 overwrites the tile
  if (tid < 64) {
#pragma unroll
    for (int i = 0; i < 16; ++i) first[i] = i < k ? ft[perm[i] * kNarrowCS + c] : cplx<T>{0, 0};
  }
  __syncthreads();
  if (tid < 64 && c < nc) {
    narrow_block<T, 16, true>(first, A, ks, nullptr, 0, 0, min(16, k), nullptr);
#pragma unroll
    for (int i = 0; i < 16; ++i)
      if (i < k) st_el(Y + i * ld + c, first[i]);
    int h = 16;
    for (; h + 16 <= k; h += 16) narrow_upper<T, 16>(A, ks, Y + c, ld, h, 16);
    if (h + 8 <= k) narrow_upper<T, 8>(A, ks, Y + c, ld, h, 8), h += 8;
    for (; h < k; h += 4) narrow_upper<T, 4>(A, ks, Y + c, ld, h, min(4, k - h));
  } else if (tid >= 64 && c < nc) {
    int h = 0;
    for (; h + 16 <= k; h += 16) narrow_lower<T, 16>(A, ks, ft + c, dinv, h, 16);
    if (h + 8 <= k) narrow_lower<T, 8>(A, ks, ft + c, dinv, h, 8), h += 8;
    for (; h < k; h += 4) narrow_lower<T, 4>(A, ks, ft + c, dinv, h, min(4, k - h));
  }
  __syncthreads();
  for (int q = wid; q < nc; q += NW)
    for (int r = lane; r < k; r += 32) st_el(F + (k + tk.c0 + q) * ld + r, ft[r * kNarrowCS + q]);
}

}  // namespace ss
