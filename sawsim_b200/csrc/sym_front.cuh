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
// Pivots are searched inside a block only; points whose factors show that (run_sweep) are
// solved again on the general path, which searches all of a front's pivot rows.
// The maps are monotone, so upper entries come from upper entries.  A front's memory
// holds, for every pivot block, L and U of F11 in pivot order, U12 right of it and L21
// below it (its rows in front order): the row interchanges of a later block are not
// applied to the L21 rows of an earlier one, the solves apply each block's interchange
// when they reach it.
#pragma once
#include <type_traits>

namespace ss {

// Upper triangle of an update block = (its sources) - L21 U12 on the FP64 tensor cores,
// in tiles of 32 x BN by four warps of 16 x BN / 2 each (three real products per complex
// 8x8x4 block, operands staged as in front_dmma3_kernel).  The sources' entries are
// copied into the staged C tile by cp.async when the CTA starts, so their latency overlaps
// the K loop; entries that both sources have take the second one in the epilogue.  Tiles
// below the diagonal are not launched; in the others a warp skips its 8x8 blocks below it,
// and the K loop its last half chunk when that is empty.
//   32 x 32, for short products: four CTAs per SM, the first operands are asked for before the
// sources' row maps, and the second source's entries with the first ones.
// Launches one at a time: 0.40 of the byte and operation bound on 16x64 ME0 (101 points, every
// update short), 0.55 on 32x128 ME1 (51 points).
//   32 x 64: 96 accumulator registers, three CTAs per SM; 0.75 of that bound on 32x128 ME1.
// 64 x 64 tiles (two CTAs) wait for C more and leave more of a diagonal tile unused: 40.2
// against 33.7 ms for the updates of the 64x256 ME1 cell at 11 points, 10.5 against 8.6 ms
// for the 8x2x26 Hex27 slab at 33.
template <int BN>
constexpr int sym_schur_smem() { return 32 * (BN + 1) * (int)sizeof(cd); }
template <int BN>
__global__ void __launch_bounds__(128, BN == 64 ? 3 : 4)
    sym_schur_kernel(FrontArgs<double> a, const GemmTask *__restrict__ tasks) {
  constexpr int MB = 2, BM = 16 * MB, WR = 8 * MB, BS = BN + 2, WC = BN / 2, NJ = WC / 8, CS = BN + 1;
  __shared__ __align__(16) cd As[2][BM * kDmmaAS];
  __shared__ __align__(16) cd Bs[2][kDmmaBK * BS];
  __shared__ int ir[2][BM], ic[2][BN];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  cd *Cs = reinterpret_cast<cd *>(smem_raw);
  const GemmTask tk = tasks[blockIdx.x];
  const SymFront &s = a.sf[tk.f];
  const int ld = s.ld, nch = s.nch;
  cd *arena = a.arena + (int64_t)blockIdx.y * a.stride;
  cd *F = arena + s.off;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int wm = wid >> 1, wn = wid & 1;
  const int g = lane >> 2, t = lane & 3;
  auto issue = [&](int buf, int kb) {
#pragma unroll
    for (int q = 0; q < BM * kDmmaBK / 128; ++q) {
      const int idx = threadIdx.x + 128 * q;
      const int r = idx / kDmmaBK, k = idx % kDmmaBK;
      const int gr = tk.r0 + r, gk = kb + k;
      const bool ok = gr < tk.rhi && gk < tk.kk1;
      cp_async16_cd((uint32_t)__cvta_generic_to_shared(&As[buf][r * kDmmaAS + dmma_acol(r, k)]),
                    ok ? F + (int64_t)gr * ld + gk : F, ok ? 16u : 0u);
    }
#pragma unroll
    for (int q = 0; q < kDmmaBK * BN / 128; ++q) {
      const int idx = threadIdx.x + 128 * q;
      const int k = idx / BN, c = idx % BN;
      const int gk = kb + k, gc = tk.c0 + c;
      const bool ok = gk < tk.kk1 && gc < tk.chi;
      cp_async16_cd((uint32_t)__cvta_generic_to_shared(&Bs[buf][k * BS + c]), ok ? F + (int64_t)gk * ld + gc : F,
                    ok ? 16u : 0u);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int nk = (tk.kk1 - tk.kk0 + kDmmaBK - 1) / kDmmaBK;
  if (BN == 32) issue(0, tk.kk0);
  if (nch) {
    sym_stage<double, BM, BN, 128, CS>(Cs, s, arena, a.imap, tk, ir, ic);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // first column block of the warp with an entry on or above the diagonal, per row block:
  // row block i needs column blocks j with 8 j + 7 >= 8 i + dr
  const int dr = tk.r0 + wm * WR - (tk.c0 + wn * WC);
  auto j0 = [&](int i) { return (8 * i + dr - 7 + 7) >> 3; };    // ceil((8 i + dr - 7) / 8)
  const int rows = min(tk.rhi, tk.r0 + BM) - (tk.r0 + wm * WR);  // the warp's rows inside the tile
  // entries that both sources have: the second source's
  cd cv[BN == 64 ? 1 : MB][NJ][2];
  auto second = [&](int i) {
    const int rl = wm * WR + i * 8 + g, r = tk.r0 + rl;
    const bool two = nch > 1 && r < tk.rhi;
    const int i0 = two ? ir[0][rl] : -1, i1 = two ? ir[1][rl] : -1;
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cl = wn * WC + j * 8 + 2 * t + e, c = tk.c0 + cl;
        cd &v = cv[BN == 64 ? 0 : i][j][e];
        v = cd{0.0, 0.0};
        if ((i0 | i1) >= 0 && c >= r && c < tk.chi && (ic[0][cl] | ic[1][cl]) >= 0)
          v = ld_once(arena + s.cb[1] + (int64_t)i1 * s.cld[1] + ic[1][cl]);
      }
  };
  if (BN == 32) {       // all of them with the first loads
#pragma unroll
    for (int i = 0; i < MB; ++i) second(i);
  }
  double p1[MB][NJ][2], p2[MB][NJ][2], p3[MB][NJ][2];
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) p1[i][j][e] = p2[i][j][e] = p3[i][j][e] = 0.0;
  const bool whole = j0(MB - 1) <= 0 && rows >= WR, some = rows > 0 && j0(0) < NJ;
  if (BN == 64) issue(0, tk.kk0);
  for (int kc = 0; kc < nk; ++kc) {
    const int buf = kc & 1;
    if (kc + 1 < nk) {
      issue(buf ^ 1, tk.kk0 + (kc + 1) * kDmmaBK);
      if (BN == 32 && kc == 0 && nch)
        asm volatile("cp.async.wait_group 2;" ::: "memory");     // the C tile may still be on its way
      else
        asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else if (BN == 32 && kc == 0 && nch) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    auto half = [&](int kk, auto whole_c) {
      constexpr bool WHOLE = decltype(whole_c)::value;
      cd av[MB];
      double as[MB];
#pragma unroll
      for (int i = 0; i < MB; ++i) {
        const int ar = wm * WR + i * 8 + g;
        av[i] = As[buf][ar * kDmmaAS + dmma_acol(ar, kk + t)];
        as[i] = av[i].x + av[i].y;
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        if (!WHOLE && j < j0(0)) continue;
        const cd bv = Bs[buf][(kk + t) * BS + wn * WC + j * 8 + g];
        const double bs = bv.x + bv.y;
#pragma unroll
        for (int i = 0; i < MB; ++i) {
          if (!WHOLE && (j < j0(i) || 8 * i >= rows)) continue;
          dmma(p1[i][j][0], p1[i][j][1], av[i].x, bv.x);
          dmma(p2[i][j][0], p2[i][j][1], av[i].y, bv.y);
          dmma(p3[i][j][0], p3[i][j][1], as[i], bs);
        }
      }
    };
    const bool second = tk.kk0 + kc * kDmmaBK + 4 < tk.kk1;
    if (whole) {
      half(0, std::true_type{});
      if (second) half(4, std::true_type{});
    } else if (some) {
      half(0, std::false_type{});
      if (second) half(4, std::false_type{});
    }
    __syncthreads();
  }
  if (BN == 32 && nk == 1 && nch) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < MB; ++i) {
    const int rl = wm * WR + i * 8 + g, r = tk.r0 + rl;
    if (r >= tk.rhi) continue;
    cd *Fr = F + (int64_t)r * ld;
    if (BN == 64) second(i);
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int cl = wn * WC + j * 8 + 2 * t + e, c = tk.c0 + cl;
        if (c < r || c >= tk.chi) continue;
        cd v = cv[BN == 64 ? 0 : i][j][e];
        if (nch) v = Cs[rl * CS + cl] + v;
        const double re = p1[i][j][e] - p2[i][j][e];
        const double im = p3[i][j][e] - p1[i][j][e] - p2[i][j][e];
        st_el(Fr + c, v - cd{re, im});
      }
  }
}

// ------------------------------------------------------------------ pivot blocks
// A pivot block takes two kernels (and the Schur update) instead of the assembly, panel
// LU, row-swap, L21, U12 and panel-GEMM launches of every 32-pivot step:
//  * sym_pivot_kernel assembles F11 in shared memory, factors it there four pivots at a
//    time (block_lu) and writes it in pivot order, its 16 x 16 diagonal blocks as
//    inverses (of the unit lower and of the upper triangle, in their places): the panel
//    kernel and the solves multiply by them instead of substituting;
//  * sym_panel_kernel takes one chunk of columns of F12: it assembles the chunk in shared
//    memory and solves it as rows of F21 = F12^T (z U11 = f^T: L21) and as columns of F12
//    (L11 y = P f: U12), 16 unknowns at a time with the inverted diagonal blocks.
// With the block's LU in shared memory, one thread per panel column and a 16-step
// substitution in the solves, a pass over the 32x128 ME1 cell at 51 points took 89 ms and
// one over 16x64 at 101 points 21 ms; so, 61 and 15 ms.
// Row interchanges are implicit (a mask of eliminated rows); `piv` receives, for each
// pivot position, the block's row it came from (the solve kernels gather).
constexpr int kDiagB = 16;        // inverted diagonal blocks

// F11 of one pivot block with its arrowhead entries [a0, a1), or (c0 >= 0) the chunk of
// F12 that starts at update column c0 with its entries
struct NarrowTask {
  int f, c0, a0, a1;
};
__host__ __device__ constexpr int pivot_class(int k) { return k <= 16 ? 16 : k <= 32 ? 32 : k <= 48 ? 48 : 64; }
__host__ __device__ constexpr int pivot_ks(int k) { return (k + 3) / 4 * 4 + 1; }   // odd: columns without conflicts
template <class T>
__host__ __device__ constexpr size_t pivot_smem(int k) {
  return (size_t)k * pivot_ks(k) * sizeof(cplx<T>) + (size_t)2 * k * sizeof(int);
}

// magnitude |x| + |y| of a pivot candidate as an ordered integer, its low 7 bits replaced by
// the row (the lowest row wins among magnitudes equal to about 2^-13)
__device__ __forceinline__ unsigned pivot_key(double v, int r) {
  return ((unsigned)__double2hiint(v) & ~127u) | (unsigned)(127 - r);
}
__device__ __forceinline__ unsigned pivot_key(float v, int r) {
  return (__float_as_uint(v) & ~127u) | (unsigned)(127 - r);
}
// l = v / z for a pivot z with its key: conj(z) v times 1 / |z|^2, z scaled by the power of
// two that brings |x| + |y| into [1, 2), so no square over- or underflows.
struct PivotRecip {
  cd z;          // conj(scaled pivot)
  double g;      // scale / |scaled pivot|^2
  __device__ __forceinline__ PivotRecip(cd p, unsigned key) {
    const double r = __hiloint2double(min(max(2046 - (int)(key >> 20), 1), 2045) << 20, 0);
    z = cd{p.x * r, -p.y * r};
    g = __drcp_rn(z.x * z.x + z.y * z.y) * r;
  }
  __device__ __forceinline__ cd recip() const { return cd{z.x * g, z.y * g}; }
  __device__ __forceinline__ cd times(cd v) const {
    const cd t = cmul(v, z);     // beside the reciprocal's chain
    return cd{t.x * g, t.y * g};
  }
};
struct PivotRecipF {
  cf z;
  float g;
  __device__ __forceinline__ PivotRecipF(cf p, unsigned key) {
    const float r = __uint_as_float(min(max(254 - (int)(key >> 23), 1), 253) << 23);
    z = cf{p.x * r, -p.y * r};
    g = __frcp_rn(z.x * z.x + z.y * z.y) * r;
  }
  __device__ __forceinline__ cf recip() const { return cf{z.x * g, z.y * g}; }
  __device__ __forceinline__ cf times(cf v) const {
    const cf t = cmul(v, z);
    return cf{t.x * g, t.y * g};
  }
};

// A warp's 16 columns (from c0) of the block that block_lu factors, in registers: in
// complex128 as accumulators of the FP64 tensor cores, in complex64 a row (KMAX > 32: two
// rows) per lane.
template <class T, int KMAX> struct LuTile;
template <int KMAX> struct LuTile<double, KMAX> {
  static constexpr int RB = KMAX / 8;
  double cr[RB][2][2], ci[RB][2][2];
  int g, t;
  __device__ __forceinline__ void load(const cd *W, int ks, int k, int c0) {
    g = (threadIdx.x & 31) >> 2;
    t = threadIdx.x & 3;
#pragma unroll
    for (int i = 0; i < RB; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int r = 8 * i + g, c = c0 + 8 * j + 2 * t + e;
          const cd z = r < k && c < k ? W[r * ks + c] : cd{0.0, 0.0};
          cr[i][j][e] = z.x;
          ci[i][j][e] = z.y;
        }
  }
  // the columns [lo, hi) of the rows in the mask to W
  __device__ __forceinline__ void put(cd *W, int ks, int c0, unsigned long long rows, int lo, int hi) const {
    rows >>= g;
    cd *Wg = W + g * ks + c0 + 2 * t;
    bool in[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = c0 + 8 * j + 2 * t + e;
        in[j][e] = c >= lo && c < hi;
      }
#pragma unroll
    for (int i = 0; i < RB; ++i)
      if (rows >> (8 * i) & 1) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e)
            if (in[j][e]) Wg[8 * i * ks + 8 * j + e] = cd{cr[i][j][e], ci[i][j][e]};
      }
  }
  // open rows -= (columns j0 .. j0 + 3 of W) (rows perm[j0 + s] of W), columns >= j0 + 4
  __device__ __forceinline__ void update(const cd *W, int ks, int k, int c0, int j0, const int *perm,
                                         unsigned long long open) {
    const cd *Wb = W + perm[j0 + t] * ks, *Wa = W + g * ks + j0 + t;
    open >>= g;
    cd b[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) b[j] = Wb[min(c0 + 8 * j + g, ks - 1)];
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      if (8 * i >= k) break;
      const cd a = open >> (8 * i) & 1 ? Wa[8 * i * ks] : cd{0.0, 0.0};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (c0 + 8 * j + 8 <= j0 + 4) continue;
        dmma(cr[i][j][0], cr[i][j][1], -a.x, b[j].x);
        dmma(ci[i][j][0], ci[i][j][1], -a.x, b[j].y);
        dmma(cr[i][j][0], cr[i][j][1], a.y, b[j].y);
        dmma(ci[i][j][0], ci[i][j][1], -a.y, b[j].x);
      }
    }
  }
};
template <int KMAX> struct LuTile<float, KMAX> {
  static constexpr int R = KMAX > 32 ? 2 : 1;
  cf v[R][16];
  int lane;
  __device__ __forceinline__ void load(const cf *W, int ks, int k, int c0) {
    lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int c = 0; c < 16; ++c)
        v[i][c] = lane + 32 * i < k && c0 + c < k ? W[(lane + 32 * i) * ks + c0 + c] : cf{0.f, 0.f};
  }
  __device__ __forceinline__ void put(cf *W, int ks, int c0, unsigned long long rows, int lo, int hi) const {
#pragma unroll
    for (int i = 0; i < R; ++i)
      if (rows >> (lane + 32 * i) & 1) {
#pragma unroll
        for (int c = 0; c < 16; ++c)
          if (c0 + c >= lo && c0 + c < hi) W[(lane + 32 * i) * ks + c0 + c] = v[i][c];
      }
  }
  __device__ __forceinline__ void update(const cf *W, int ks, int k, int c0, int j0, const int *perm,
                                         unsigned long long open) {
    cf l[R][4];
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int s = 0; s < 4; ++s)
        l[i][s] = open >> (lane + 32 * i) & 1 ? W[(lane + 32 * i) * ks + j0 + s] : cf{0.f, 0.f};
    const cf *Wc[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) Wc[s] = W + perm[j0 + s] * ks + c0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (c0 + 4 * q < j0 + 4 || c0 + 4 * q >= k) continue;
#pragma unroll
      for (int c = 4 * q; c < 4 * q + 4; ++c)
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const cf u = Wc[s][c];
#pragma unroll
          for (int i = 0; i < R; ++i) v[i][c] = cfms(v[i][c], l[i][s], u);
        }
    }
  }
};

// LU of the k x k matrix W (row stride ks, shared memory; k <= KMAX) in place with
// implicit row interchanges, by KMAX / 16 warps with 16 columns each in registers.  Four
// columns at a time: their warp puts them into W, eliminates them with a row in each lane's
// registers (the pivot by one integer reduction of candidate keys) and leaves the
// multipliers there; then every warp with columns left takes its entries of the four pivot
// rows through a 4 x 4 triangle and subtracts the rank-4 product.  One barrier per four
// pivots, and a pivot's chain is one warp's; the next four columns start as soon as their
// own warp has applied the last ones.
//   Bound by the chain of a pivot (about 18 dependent FP64 operations of some 20 cycles,
// one reduction, two trips through shared memory: 1100 cycles).  12 launches of one to ten
// 48-pivot blocks (16x64 ME0, one point): 0.59 ms, against 0.69 with two threads per row and
// a block-wide step per pivot; the 89 wide complex64 launches of the 12x4x48 slab: 4.0
// against 6.1 ms.  On return W holds the multipliers and U rows in
// the original row order, perm[j] the row of pivot j and dinv[j] the reciprocal pivots.
template <class T, int KMAX>
__device__ __forceinline__ int block_lu(cplx<T> *W, int ks, int k, T tiny, int *perm, cplx<T> *dinv) {
  constexpr int R = KMAX > 32 ? 2 : 1;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, c0 = 16 * wid;
  LuTile<T, KMAX> tile;
  tile.load(W, ks, k, c0);
  unsigned long long open = k < 64 ? (1ull << k) - 1 : ~0ull;     // rows without a pivot
  int npert = 0;
  for (int j0 = 0; j0 < k; j0 += 4) {
    if (wid == j0 >> 4) {
      tile.put(W, ks, c0, open, j0, j0 + 4);
      __syncwarp();
      cplx<T> v[R][4];
      bool op[R];
#pragma unroll
      for (int i = 0; i < R; ++i) {
        const int r = lane + 32 * i;
        op[i] = open >> r & 1;
#pragma unroll
        for (int s = 0; s < 4; ++s) v[i][s] = op[i] ? W[r * ks + j0 + s] : cplx<T>{0, 0};
      }
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        if (j0 + s >= k) break;
        unsigned key = 0u;
#pragma unroll
        for (int i = 0; i < R; ++i)
          if (op[i]) key = max(key, pivot_key(cabs1(v[i][s]), lane + 32 * i));
        key = __reduce_max_sync(0xffffffffu, key);
        const int p = 127 - (int)(key & 127u);
        cplx<T> *Wp = W + p * ks + j0;
        if ((key | 127u) <= (pivot_key(tiny, 0) | 127u)) {      // at most about tiny
#pragma unroll
          for (int i = 0; i < R; ++i)
            if (p == lane + 32 * i && cabs1(v[i][s]) < tiny) {
              v[i][s] = cplx<T>{tiny, (T)0};
              ++npert;
            }
          key = pivot_key(tiny, 0);
        }
#pragma unroll
        for (int i = 0; i < R; ++i)
          if (p == lane + 32 * i) {
#pragma unroll
            for (int c = s; c < 4; ++c) Wp[c] = v[i][c];
            perm[j0 + s] = p;
            op[i] = false;
          }
        __syncwarp();
        const std::conditional_t<sizeof(T) == 8, PivotRecip, PivotRecipF> rec(Wp[s], key);
#pragma unroll
        for (int i = 0; i < R; ++i) {
          const cplx<T> l = rec.times(v[i][s]);
          if (!op[i]) continue;
          W[(lane + 32 * i) * ks + j0 + s] = l;
#pragma unroll
          for (int c = s + 1; c < 4; ++c) v[i][c] = cfms(v[i][c], l, Wp[c]);
        }
        if (lane == 0) dinv[j0 + s] = rec.recip();
      }
    }
    __syncthreads();
    if (j0 + 4 >= k) break;
    int p[4];
    unsigned long long taken = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      p[s] = perm[j0 + s];
      taken |= 1ull << p[s];
    }
    open &= ~taken;
    if (c0 >= k || c0 + 16 <= j0 + 4) continue;
    // the warp's columns of the pivot rows
    tile.put(W, ks, c0, taken, j0 + 4, ks - 1);
    __syncwarp();
    const int c = c0 + lane;
    if (lane < 16 && c >= j0 + 4 && c < ks - 1) {
      cplx<T> u[4];
#pragma unroll
      for (int s = 0; s < 4; ++s) u[s] = W[p[s] * ks + c];
#pragma unroll
      for (int s = 1; s < 4; ++s) {
#pragma unroll
        for (int q = 0; q < s; ++q) u[s] = cfms(u[s], W[p[s] * ks + j0 + q], u[q]);
        W[p[s] * ks + c] = u[s];
      }
    }
    __syncwarp();
    tile.update(W, ks, k, c0, j0, perm, open);
  }
  return npert;
}

// (In complex128 with KMAX = 64 the 168 registers of three CTAs per SM spill 228 bytes of
// stores and 276 of loads per thread.)
template <class T, int KMAX>
__global__ void __launch_bounds__(2 * KMAX, KMAX == 64 ? 3 : KMAX == 48 ? 4 : KMAX == 32 ? 8 : 12)
    sym_pivot_kernel(FrontArgs<T> a, const NarrowTask *__restrict__ tasks, int nb, const uint16_t *__restrict__ apos,
                     const int *__restrict__ aslot) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ cplx<T> dinv[KMAX];
  __shared__ int perm[KMAX];
  constexpr int NT = 2 * KMAX, NW = NT / 32;
  const NarrowTask tk = tasks[blockIdx.x / nb];
  const int fq = blockIdx.x % nb;
  const SymFront &s = a.sf[tk.f];
  const int k = s.k, ks = pivot_ks(k);
  cplx<T> *W = reinterpret_cast<cplx<T> *>(smem_raw);
  int *ir = reinterpret_cast<int *>(W + k * ks);
  cplx<T> *arena = a.arena + (int64_t)fq * a.stride;
  const double om = a.omega[fq];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nch = s.nch;
  // a load is a round trip of 1000 to 2000 cycles here: few of them in a row, many at once
  Arrows<T, 2> arrows;
  arrows.index(tk.a0, tk.a1, apos, aslot);
  if (nch) {
    for (int i = tid; i < k; i += NT) {
      ir[i] = a.imap[s.imap[0] + i];
      ir[k + i] = nch > 1 ? a.imap[s.imap[1] + i] : -1;
    }
    arrows.load(a);
    __syncthreads();
    // the sources' upper entries, mirrored: eight rows of 32 columns in flight per warp
    constexpr int U = 8;
    for (int cb = 0; cb < k; cb += 32)
      for (int rb = wid; rb < min(k, cb + 32); rb += U * NW) {
        const int c = cb + lane, cc = min(c, k - 1);
        cplx<T> v0[U], v1[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int r = rb + u * NW, rr = min(r, k - 1);
          sym_pick<T>(s, arena, r < k && c < k && c >= r, ir[rr], ir[cc], ir[k + rr], ir[k + cc], v0[u], v1[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int r = rb + u * NW;
          if (r < k && c < k && c >= r) {
            const cplx<T> v = v0[u] + v1[u];
            W[r * ks + c] = v;
            W[c * ks + r] = v;
          }
        }
      }
  } else {
    arrows.load(a);
    for (int t = tid; t < k * ks; t += NT) W[t] = cplx<T>{0, 0};
  }
  __syncthreads();
  arrows.add_all(a, tk.a0, tk.a1, apos, aslot, om, [&](int p, cplx<T> e) {
    const int r = p >> 6, c = p & 63;
    const cplx<T> v = W[r * ks + c] + e;
    W[r * ks + c] = v;
    W[c * ks + r] = v;
  });
  __syncthreads();
  const int np = block_lu<T, KMAX>(W, ks, k, a.tiny, perm, dinv);
  if (np) atomicAdd(a.nperturb + fq, np);
  cplx<T> *F = arena + s.off;
  const int ld = s.ld;
  for (int r = wid; r < k; r += NW) {
    const cplx<T> *row = W + perm[r] * ks;
    for (int c = lane; c < k; c += 32)
      if ((c ^ r) >= kDiagB) st_el(F + (int64_t)r * ld + c, row[c]);
  }
  for (int i = tid; i < k; i += NT) a.piv[(int64_t)fq * a.n + s.p0 + i] = perm[i];
  // inverses of the diagonal blocks, one block per warp: lanes 0-15 a column of the
  // inverted unit lower triangle each, lanes 16-31 of the inverted upper triangle with its
  // rows and columns in reverse order, so that both halves run the same substitution
  const int h0 = kDiagB * wid, hw = min(kDiagB, k - h0);
  if (hw <= 0) return;
  const bool upper = lane >= 16;
  const int col = lane & 15;                   // the column, counted as the rows are
  const int first = h0 + (upper ? hw - 1 : 0), dir = upper ? -1 : 1;
  cplx<T> x[kDiagB];
#pragma unroll
  for (int i = 0; i < kDiagB; ++i) x[i] = cplx<T>{i == col ? (T)1 : (T)0, (T)0};
#pragma unroll
  for (int q = 0; q < kDiagB; ++q) {
    if (q >= hw) break;
    const int r = first + dir * q;
    if (upper) x[q] = cmul(x[q], dinv[r]);
    if ((upper ? q >= col : q > col) && col < hw) st_el(F + (int64_t)r * ld + first + dir * col, x[q]);
#pragma unroll
    for (int i = q + 1; i < kDiagB; ++i)
      if (i < hw) x[i] = cfms(x[i], W[perm[first + dir * i] * ks + r], x[q]);
  }
}

// ------------------------------------------------------------------ panel columns
// Coefficient (i, t) of an inverted diagonal block at A (row stride ks): LOWER the unit
// lower triangle's inverse, else the transposed inverse of the upper triangle (both are
// lower triangular in (i, t)).
template <class T, bool LOWER>
__device__ __forceinline__ cplx<T> diag_coef(const cplx<T> *A, int ks, int i, int t) {
  if (t > i) return cplx<T>{0, 0};
  if (LOWER && t == i) return cplx<T>{1, 0};
  return LOWER ? A[i * ks + t] : A[t * ks + i];
}

// complex128: 8 MB columns of the chunk (from cb) solved by one warp as 8 MB rows of the
// transposed system, U12^T L11^T = (P F12)^T (LOWER) or L21 U11 = F12^T, on the FP64 tensor
// cores.  The rows stay in accumulator registers; 16 pivots at a time they are multiplied
// by the inverted diagonal block, written out, and subtracted from the columns to the
// right (three real products per complex 8x8x4 block); an accumulator becomes the next
// product's operand by shuffles within four lanes.
template <bool LOWER, int KB, int MB>
__device__ __forceinline__ void panel_dmma(const cd *A, int ks, const cd *Y, int CS, const int *perm, int k, int cb,
                                           int nc, cd *out, int64_t ld) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, nbk = (k + 7) >> 3;
  double xr[MB][KB][2], xi[MB][KB][2];
#pragma unroll
  for (int j = 0; j < KB; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = 8 * j + 2 * t + e;
      const int row = j < nbk ? (LOWER ? perm[r] : r) : 0;
#pragma unroll
      for (int b = 0; b < MB; ++b) {
        const cd z = j < nbk ? Y[row * CS + cb + 8 * b + g] : cd{0.0, 0.0};
        xr[b][j][e] = z.x;
        xi[b][j][e] = z.y;
      }
    }
  // columns 4 h + t of an 8-column block held as columns 2 t, 2 t + 1
  auto turn = [&](const double (&x)[2], int h) {
    const int src = (lane & ~3) | (2 * h + (t >> 1));
    const double x0 = __shfl_sync(0xffffffffu, x[0], src), x1 = __shfl_sync(0xffffffffu, x[1], src);
    return t & 1 ? x1 : x0;
  };
  double ar[MB][2][2], ai[MB][2][2];      // operand: two 8-column blocks of two steps
  auto operand = [&](int j, int kb) {
#pragma unroll
    for (int b = 0; b < MB; ++b)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ar[b][kb][h] = turn(xr[b][j], h);
        ai[b][kb][h] = turn(xi[b][j], h);
      }
  };
  double p[MB][3][2];
  auto clear = [&] {
#pragma unroll
    for (int b = 0; b < MB; ++b)
#pragma unroll
      for (int q = 0; q < 3; ++q) p[b][q][0] = p[b][q][1] = 0.0;
  };
  auto mma = [&](int kb, int h, cd bv) {
    const double bs = bv.x + bv.y;
#pragma unroll
    for (int b = 0; b < MB; ++b) {
      dmma(p[b][0][0], p[b][0][1], ar[b][kb][h], bv.x);
      dmma(p[b][1][0], p[b][1][1], ai[b][kb][h], bv.y);
      dmma(p[b][2][0], p[b][2][1], ar[b][kb][h] + ai[b][kb][h], bs);
    }
  };
#pragma unroll
  for (int q = 0; q < (KB + 1) / 2; ++q) {
    if (2 * q >= nbk) break;
    const cd *D = A + 16 * q * (ks + 1);
    const int nb2 = min(2, nbk - 2 * q);         // 8-column blocks of this diagonal block
    operand(2 * q, 0);
    if (2 * q + 1 < KB && nb2 > 1) operand(2 * q + 1, 1);
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      if (2 * q + n >= KB || n >= nb2) break;
      clear();
#pragma unroll
      for (int kb = 0; kb <= n; ++kb)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int kk = 8 * kb + 4 * h + t, nn = 8 * n + g;
          cd bv = LOWER ? D[nn * ks + kk] : D[kk * ks + nn];
          if (kb == n) {
            if (kk > nn) bv = cd{0.0, 0.0};
            if (LOWER && kk == nn) bv = cd{1.0, 0.0};
          }
          mma(kb, h, bv);
        }
      const int j = 2 * q + n;
#pragma unroll
      for (int b = 0; b < MB; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double re = p[b][0][e] - p[b][1][e], im = p[b][2][e] - p[b][0][e] - p[b][1][e];
          xr[b][j][e] = re;
          xi[b][j][e] = im;
          const int c = cb + 8 * b + g, r = 8 * j + 2 * t + e;
          if (c < nc && r < k) st_el(LOWER ? out + r * ld + c : out + c * ld + r, cd{re, im});
        }
    }
    if (2 * q + 2 >= KB || 2 * q + 2 >= nbk) break;
    operand(2 * q, 0);
    operand(2 * q + 1, 1);
#pragma unroll
    for (int n = 2 * q + 2; n < KB; ++n) {
      if (n >= nbk) break;
      clear();
#pragma unroll
      for (int kb = 0; kb < 2; ++kb)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int kk = 16 * q + 8 * kb + 4 * h + t, nn = 8 * n + g;
          mma(kb, h, LOWER ? A[nn * ks + kk] : A[kk * ks + nn]);
        }
#pragma unroll
      for (int b = 0; b < MB; ++b)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          xr[b][n][e] -= p[b][0][e] - p[b][1][e];
          xi[b][n][e] -= p[b][2][e] - p[b][0][e] - p[b][1][e];
        }
    }
  }
}

// complex64: 16 columns of the tile solved in place by one warp, 16 rows at a time: a
// lane holds 4 rows x 2 columns, so each coefficient and each solved entry it loads takes
// part in two and four multiply-adds (one column per thread is bound by the broadcast
// loads).
template <bool LOWER>
__device__ __forceinline__ void panel_simt(const cf *A, int ks, cf *Y, int CS, int k) {
  const int lane = threadIdx.x & 31, c = 2 * (lane & 7), r = 4 * (lane >> 3);
  for (int h0 = 0; h0 < k; h0 += kDiagB) {
    cf x[4][2];
    auto load = [&](cf (&y)[2], int row) {
      const float4 q = *reinterpret_cast<const float4 *>(Y + row * CS + c);
      y[0] = cf{q.x, q.y};
      y[1] = cf{q.z, q.w};
    };
    auto store = [&](int row, const cf (&y)[2]) {
      *reinterpret_cast<float4 *>(Y + row * CS + c) = make_float4(y[0].x, y[0].y, y[1].x, y[1].y);
    };
    if (h0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) load(x[i], h0 + r + i);
#pragma unroll 4
      for (int t = 0; t < h0; ++t) {
        cf y[2];
        load(y, t);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const cf q = LOWER ? A[(h0 + r + i) * ks + t] : A[t * ks + h0 + r + i];
          x[i][0] = cfms(x[i][0], q, y[0]);
          x[i][1] = cfms(x[i][1], q, y[1]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) store(h0 + r + i, x[i]);
      __syncwarp();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i][0] = x[i][1] = cf{0.f, 0.f};
#pragma unroll 4
    for (int t = 0; t < kDiagB; ++t) {
      cf y[2];
      load(y, h0 + t);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const cf q = diag_coef<float, LOWER>(A + h0 * ks + h0, ks, r + i, t);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          x[i][e].x = fmaf(q.x, y[e].x, fmaf(-q.y, y[e].y, x[i][e].x));
          x[i][e].y = fmaf(q.x, y[e].y, fmaf(q.y, y[e].x, x[i][e].y));
        }
      }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 4; ++i) store(h0 + r + i, x[i]);
    __syncwarp();
  }
}

// Four warps for L21 and four for U12 of the same chunk.  (Four warps that solved one after
// the other, with P F12 through global memory: 45.5 against 42.6 ms for the factorisation of
// the 32x128 ME1 cell at 51 points, where complex128 keeps its rows in registers too.)  In
// complex128 with 64 columns the 128 registers of two CTAs per SM spill 264 bytes of stores
// and 292 of loads per thread.  Launches one at a time: 6.8 ms for the 64-column chunks of that
// sweep and 6.6 for the 32-column ones, 3.4 and 2.6 times what their bytes or operations take.
constexpr int kPanelThreadsSym = 256;
// chunk width and padded sizes: the tile and F11 of one chunk leave room for at least two
// CTAs per SM (complex128, 64 pivots: 104 KB at 32 columns; 64 would take 137)
template <class T>
__host__ __device__ constexpr int panel_cols(int k) {
  return sizeof(T) == 8 && k > 40 ? 32 : 64;
}
template <class T>
__host__ __device__ constexpr int panel_rows(int k) {
  return sizeof(T) == 8 ? (k + 7) / 8 * 8 : (k + 15) / 16 * 16;
}
template <class T>
__host__ __device__ constexpr int panel_ks(int k) {
  return panel_rows<T>(k) + (sizeof(T) == 8 ? 4 : 1);
}
template <class T>
__host__ __device__ constexpr size_t panel_smem(int k, int cw) {
  // (complex64 solves L21 and U12 in tiles of their own)
  return ((size_t)panel_rows<T>(k) * (panel_ks<T>(k) + (sizeof(T) == 8 ? 1 : 2) * (cw + 2))) * sizeof(cplx<T>) +
         (size_t)panel_rows<T>(k) * sizeof(int);
}

template <class T, int CW>
__global__ void __launch_bounds__(kPanelThreadsSym, 2)
    sym_panel_kernel(FrontArgs<T> a, const NarrowTask *__restrict__ tasks, int nb, const uint16_t *__restrict__ apos,
                     const int *__restrict__ aslot) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int NT = kPanelThreadsSym, NW = NT / 32, CS = CW + 2, NH = CW / 32;
  const NarrowTask tk = tasks[blockIdx.x / nb];
  const int fq = blockIdx.x % nb;
  const SymFront &s = a.sf[tk.f];
  const int k = s.k, kp = panel_rows<T>(k), ks = panel_ks<T>(k), nc = min(CW, s.m - k - tk.c0);
  const int64_t ld = s.ld;
  cplx<T> *A = reinterpret_cast<cplx<T> *>(smem_raw);   // F11 in pivot order, zero past k
  cplx<T> *Y = A + kp * ks;                             // the chunk
  int *perm = reinterpret_cast<int *>(Y + (sizeof(T) == 8 ? 1 : 2) * kp * CS);
  cplx<T> *arena = a.arena + (int64_t)fq * a.stride;
  cplx<T> *F = arena + s.off;
  const double om = a.omega[fq];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int nch = s.nch;
  Arrows<T, 2> arrows;
  {
    const int64_t m0 = s.imap[0], m1 = s.imap[1];
    int j0[NH], j1[NH];
    arrows.index(tk.a0, tk.a1, apos, aslot);
#pragma unroll
    for (int h = 0; h < NH; ++h) {
      const int c = lane + 32 * h;
      j0[h] = nch > 0 && c < nc ? a.imap[m0 + k + tk.c0 + c] : -1;
      j1[h] = nch > 1 && c < nc ? a.imap[m1 + k + tk.c0 + c] : -1;
    }
    arrows.load(a);
    constexpr int U = 4;
    for (int rb = wid; rb < kp; rb += U * NW) {
      cplx<T> v0[U][NH], v1[U][NH], d[U][2];
      int i0[U], i1[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = rb + u * NW;
        i0[u] = nch > 0 && r < k ? a.imap[m0 + r] : -1;
        i1[u] = nch > 1 && r < k ? a.imap[m1 + r] : -1;
        // F11 (at most 64 columns; the padding is zero)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = lane + 32 * h;
          d[u][h] = r < k && c < k ? ld_el(F + r * ld + c) : cplx<T>{0, 0};
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int h = 0; h < NH; ++h) sym_pick<T>(s, arena, true, i0[u], j0[h], i1[u], j1[h], v0[u][h], v1[u][h]);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = rb + u * NW;
        if (r >= kp) break;
#pragma unroll
        for (int h = 0; h < NH; ++h) Y[r * CS + lane + 32 * h] = v0[u][h] + v1[u][h];
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (lane + 32 * h < ks) A[r * ks + lane + 32 * h] = d[u][h];
        if (lane + 64 < ks) A[r * ks + lane + 64] = cplx<T>{0, 0};
      }
    }
    for (int i = tid; i < kp; i += NT) perm[i] = i < k ? a.piv[(int64_t)fq * a.n + s.p0 + i] : i;
  }
  __syncthreads();
  arrows.add_all(a, tk.a0, tk.a1, apos, aslot, om, [&](int p, cplx<T> e) {
    cplx<T> *d = Y + (p >> 6) * CS + (p & 63);
    *d = *d + e;
  });
  __syncthreads();
  if constexpr (sizeof(T) == 8) {
    constexpr int MB = CW / 32, KB = CW == 64 ? 5 : 8;
    const int cb = (wid & 3) * 8 * MB;
    if (cb >= nc) return;
    if (wid < 4)
      panel_dmma<false, KB, MB>(A, ks, Y, CS, perm, k, cb, nc, F + (k + tk.c0) * ld, ld);
    else
      panel_dmma<true, KB, MB>(A, ks, Y, CS, perm, k, cb, nc, F + k + tk.c0, ld);
  } else {
    // P F12 in a tile of its own; each warp on its own columns of one of the tiles
    constexpr int WC = CW / 4;
    cplx<T> *Z = Y + kp * CS;
    for (int r = wid; r < kp; r += NW)
#pragma unroll
      for (int h = 0; h < NH; ++h) Z[r * CS + lane + 32 * h] = Y[perm[r] * CS + lane + 32 * h];
    __syncthreads();
    const int cb = (wid & 3) * WC;
    if (cb >= nc) return;
    if (wid < 4) {
      panel_simt<false>(A, ks, Y + cb, CS, k);
      for (int q = 0; q < WC; ++q)
        if (cb + q < nc)
          for (int r = lane; r < k; r += 32) st_el(F + (k + tk.c0 + cb + q) * ld + r, Y[r * CS + cb + q]);
    } else {
      panel_simt<true>(A, ks, Z + cb, CS, k);
      const int c = lane % WC;
      for (int r = lane / WC; r < k; r += 32 / WC)
        if (cb + c < nc) st_el(F + r * ld + k + tk.c0 + cb + c, Z[r * CS + cb + c]);
    }
  }
}

}  // namespace ss
