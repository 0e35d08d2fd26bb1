// Symmetric scaling of the condensed system and the check that it is symmetric.
//
// The reference scales the mechanical equations by a constant s and leaves the
// electrical coupling K_uphi unscaled (piezo_fem.py:352-366, saw3d/assembly.py:300-327),
// so A_ij t_j = A_ji t_i with t = 1 on displacement DOFs and t = s on potential DOFs.
// Potential DOFs are told by their zero mass diagonal and s is the least-squares ratio
// of K_phiu to K_uphi, so assembled matrices of unknown origin need no more input than
// a mesh does.  With A T symmetric, d scales rows and t d columns (Ruiz iterations on
// the symmetric A T); the result is checked entry by entry, and a system that is not
// symmetric (an anisotropic PML on a Hex27 slab, a caller's own matrices) keeps the
// general scaling and the general fronts.
#pragma once

namespace ss {

// slot of (R, C) in a CSR row, -1 when absent
__device__ __forceinline__ int64_t csr_find(const int64_t *__restrict__ rp, const int64_t *__restrict__ ci, int64_t R,
                                            int64_t C) {
  int64_t b = rp[R], e = rp[R + 1];
  const int64_t hi = e;
  while (b < e) {
    const int64_t mid = (b + e) / 2;
    if (ci[mid] < C) b = mid + 1; else e = mid;
  }
  return b < hi && ci[b] == C ? b : -1;
}

// phi[R] = 1 on rows without mass
__global__ void sym_phi_kernel(int64_t n, const int64_t *__restrict__ rp, const int64_t *__restrict__ ci,
                               const cd *__restrict__ M, unsigned char *__restrict__ phi) {
  const int64_t R = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (R >= n) return;
  const int64_t s = csr_find(rp, ci, R, R);
  phi[R] = s < 0 || (M[s].x == 0.0 && M[s].y == 0.0);
}

// partial sums of Re(conj(K_ij) K_ji) and |K_ij|^2 over displacement rows i and
// potential columns j: warp per row, fixed-order trees (part[2 b], part[2 b + 1])
__global__ void __launch_bounds__(256) sym_ratio_kernel(int64_t n, const int64_t *__restrict__ rp,
                                                        const int64_t *__restrict__ ci, const cd *__restrict__ K,
                                                        const unsigned char *__restrict__ phi,
                                                        double *__restrict__ part) {
  __shared__ double s_a[256], s_b[256];
  const int lane = threadIdx.x & 31;
  double sa = 0.0, sb = 0.0;
  for (int64_t R = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); R < n; R += (int64_t)gridDim.x * 8) {
    if (phi[R]) continue;
    for (int64_t t = rp[R] + lane; t < rp[R + 1]; t += 32) {
      const int64_t C = ci[t];
      if (!phi[C]) continue;
      const cd v = K[t];
      if (v.x == 0.0 && v.y == 0.0) continue;
      const int64_t q = csr_find(rp, ci, C, R);
      if (q < 0) continue;
      const cd u = K[q];
      sa += v.x * u.x + v.y * u.y;
      sb += v.x * v.x + v.y * v.y;
    }
  }
  s_a[threadIdx.x] = sa;
  s_b[threadIdx.x] = sb;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      s_a[threadIdx.x] += s_a[threadIdx.x + s];
      s_b[threadIdx.x] += s_b[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) part[2 * blockIdx.x] = s_a[0], part[2 * blockIdx.x + 1] = s_b[0];
}

// t[R] from the summed ratio (1 when there is no coupling), d[R] = 1
__global__ void __launch_bounds__(256) sym_factor_kernel(int64_t n, int nparts, const double *__restrict__ part,
                                                         const unsigned char *__restrict__ phi, double *__restrict__ t,
                                                         double *__restrict__ d) {
  __shared__ double ratio;
  if (threadIdx.x == 0) {
    double sa = 0.0, sb = 0.0;
    for (int i = 0; i < nparts; ++i) sa += part[2 * i], sb += part[2 * i + 1];
    const double r = sb > 0.0 ? sa / sb : 1.0;
    ratio = r > 0.0 && isfinite(r) ? r : 1.0;
  }
  __syncthreads();
  for (int64_t R = (int64_t)blockIdx.x * 256 + threadIdx.x; R < n; R += (int64_t)gridDim.x * 256) {
    t[R] = phi[R] ? ratio : 1.0;
    d[R] = 1.0;
  }
}

// one symmetric Ruiz step on |K T| + w2 |M T| (+ wb |D T|): warp per row
__global__ void __launch_bounds__(256) sym_ruiz_kernel(int64_t n, const int64_t *__restrict__ rp,
                                                       const int64_t *__restrict__ ci, const cd *__restrict__ K,
                                                       const cd *__restrict__ M, const cd *__restrict__ D, double w2,
                                                       double wb, const double *__restrict__ t,
                                                       const double *__restrict__ d, double *__restrict__ out) {
  const int64_t R = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (R >= n) return;
  double m = 0.0;
  for (int64_t q = rp[R] + lane; q < rp[R + 1]; q += 32) {
    const int64_t c = ci[q];
    double v = sqrt(cabs2(K[q])) + w2 * sqrt(cabs2(M[q]));
    if (D) v += wb * sqrt(cabs2(D[q]));
    m = fmax(m, v * (t[c] * d[c]));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) {
    const double dr = d[R];
    out[R] = m > 0.0 ? dr / sqrt(m * dr) : dr;
  }
}

// column scale t d
__global__ void sym_cols_kernel(int64_t n, const double *__restrict__ t, const double *__restrict__ d,
                                double *__restrict__ cs) {
  const int64_t R = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (R < n) cs[R] = t[R] * d[R];
}

// asym: the largest |K'_ij - K'_ji| + w2 |M'_ij - M'_ji| (+ wb |D'|) over the scaled entry
// pairs, entries without a mirrored slot against zero, as the bits of a double (they order as
// the non-negative numbers do; infinite where a difference is not a number)
__global__ void __launch_bounds__(256) sym_check_kernel(int64_t n, const int64_t *__restrict__ rp,
                                                        const int64_t *__restrict__ ci, const cd *__restrict__ K,
                                                        const cd *__restrict__ M, const cd *__restrict__ D, double w2,
                                                        double wb, unsigned long long *__restrict__ asym) {
  const int64_t R = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (R >= n) return;
  double worst = 0.0;
  for (int64_t q = rp[R] + lane; q < rp[R + 1]; q += 32) {
    const int64_t C = ci[q];
    if (C == R) continue;
    const int64_t p = csr_find(rp, ci, C, R);
    if (p >= 0 && C < R) continue;        // the pair is checked from its upper entry
    const cd z{0.0, 0.0};
    double e = sqrt(cabs2(K[q] - (p >= 0 ? K[p] : z))) + w2 * sqrt(cabs2(M[q] - (p >= 0 ? M[p] : z)));
    if (D) e += wb * sqrt(cabs2(D[q] - (p >= 0 ? D[p] : z)));
    worst = fmax(worst, e == e ? e : INFINITY);
  }
  for (int o = 16; o > 0; o >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
  const unsigned long long bits = (unsigned long long)__double_as_longlong(worst);
  if (lane == 0 && bits > *asym) atomicMax(asym, bits);
}

}  // namespace ss
