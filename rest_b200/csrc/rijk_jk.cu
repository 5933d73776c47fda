// RI J/K kernels on the tile-packed fitted tensor (FP64 plain form).
//
// J (REST vj_upper_with_ri_v_sync / vj_upper_with_rimatr_v_sync,
// src/scf_io/mod.rs:2428-2561) is HBM-bound and runs as two streaming passes:
//   pass 1  w_P = sum_k B[P,k] W[k]   (W = D folded into the tile layout)
//   pass 2  J_k = sum_P B[P,k] w_P    (split over P, partials reduced in order)
// K (vk_upper_with_ri_v_sync, :2758-2834; dm forms :2640-2756) is a batched
// half-transform X_P = B_P C followed by a split-k rank update K = sum_P X_P X_P^T
// over 128x128 blocks of K: here on the FP64 tensor cores (DMMA), which small
// molecules use, in rijk_i8.cu on the INT8 ones.
#include <math.h>

#include <algorithm>

#include "rijk_dmma.cuh"
#include "rijk_internal.h"

namespace rijk {

Geom make_geom(int64_t n, int64_t naux) {
  Geom g;
  g.n = n;
  g.naux = naux;
  g.nt = (n + TS - 1) / TS;
  g.ntp = g.nt * (g.nt + 1) / 2;
  g.ldB = g.ntp * TILE_ELEMS;
  g.npair = n * (n + 1) / 2;
  return g;
}

static inline int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }
static inline int64_t round_up(int64_t a, int64_t b) { return cdiv(a, b) * b; }

// Largest J with J (J + 1) / 2 <= t.
__device__ __forceinline__ int64_t tri_root(int64_t t) {
  int64_t j = (int64_t)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while (j * (j + 1) / 2 > t) --j;
  while ((j + 1) * (j + 2) / 2 <= t) ++j;
  return j;
}

// ============================================================================
// layout conversion
// ============================================================================
// One CTA per stored tile (blockIdx.x), aux rows strided over blockIdx.y.
// src_kind 0: rimatr rows (npair each); 1: ri3fn blocks (n*n each).
// bmax (zeroed by the caller) or null: bmax[p ldx + mu] takes the high word of the
// largest |B_p[mu, :]|, from the elements in registers: 46 aux rows of n = 1200 take 132 us
// without, 139 with, some 500 where a pass of its own reads them back.
__global__ void __launch_bounds__(256) k_pack(int64_t n, int64_t npair, int64_t ldB, const double* __restrict__ src,
                                              int src_kind, int64_t np, double* __restrict__ dst,
                                              int* __restrict__ bmax, int64_t ldx) {
  __shared__ int m[2 * TS];  // the tile's rows, then its columns
  const int64_t t = blockIdx.x;
  const int64_t J = tri_root(t), I = t - J * (J + 1) / 2;
  const int tid = threadIdx.x;
  for (int64_t p = blockIdx.y; p < np; p += gridDim.y) {
    int row = 0;
    if (bmax) {
      __syncthreads();  // m of the aux row before is read
      if (tid < 2 * TS) m[tid] = 0;
      __syncthreads();
    }
    for (int e = tid; e < TILE_ELEMS; e += 256) {
      const int r = e & 31, c = e >> 5;
      const int64_t mu = I * TS + r, nu = J * TS + c;
      double v = 0.0;
      if (mu < n && nu < n) {
        const int64_t i = mu < nu ? mu : nu, j = mu < nu ? nu : mu;
        v = src_kind == 0 ? src[p * npair + packed_upper_index(i, j)] : src[p * n * n + i + n * j];
      }
      dst[p * ldB + t * TILE_ELEMS + e] = v;
      if (bmax) {
        const int h = __double2hiint(v) & 0x7fffffff;
        row = max(row, h);
        const int col = __reduce_max_sync(0xffffffffu, h);
        if (r == 0) m[TS + c] = col;  // a warp has a column to itself
      }
    }
    if (bmax) {
      atomicMax(&m[tid & 31], row);
      __syncthreads();
      // (a diagonal tile holds both triangles: its rows are enough)
      if (tid < (I == J ? TS : 2 * TS) && m[tid] > 0)
        atomicMax(bmax + p * ldx + (tid < TS ? I * TS + tid : J * TS + tid - TS), m[tid]);
    }
  }
}

__global__ void __launch_bounds__(256) k_unpack_rimatr(int64_t n, int64_t npair, int64_t ldB,
                                                       const double* __restrict__ src, int64_t np,
                                                       double* __restrict__ dst) {
  for (int64_t p = blockIdx.y; p < np; p += gridDim.y) {
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < npair; t += (int64_t)gridDim.x * blockDim.x) {
      const int64_t j = tri_root(t), i = t - j * (j + 1) / 2;
      const int64_t tile = tile_pair_index(i / TS, j / TS);
      dst[p * npair + t] = src[p * ldB + tile * TILE_ELEMS + (i % TS) + TS * (j % TS)];
    }
  }
}

void launch_pack(const Geom& g, const double* src, int src_kind, int64_t np, double* dst, int* bmax, int64_t ldx,
                 cudaStream_t st) {
  if (np <= 0) return;
  dim3 grid((unsigned)g.ntp, (unsigned)std::min<int64_t>(np, 65535));
  if (bmax) cudaMemsetAsync(bmax, 0, (size_t)np * ldx * sizeof(int), st);
  count_launch();
  k_pack<<<grid, 256, 0, st>>>(g.n, g.npair, g.ldB, src, src_kind, np, dst, bmax, ldx);
}
void launch_unpack_rimatr(const Geom& g, const double* src, int64_t np, double* dst, cudaStream_t st) {
  if (np <= 0) return;
  dim3 grid((unsigned)std::min<int64_t>(cdiv(g.npair, 256), 4096), (unsigned)std::min<int64_t>(np, 65535));
  count_launch();
  k_unpack_rimatr<<<grid, 256, 0, st>>>(g.n, g.npair, g.ldB, src, np, dst);
}

// ============================================================================
// failure detection
// ============================================================================
// Thread 0 initialises an mbarrier that expects one arrival and then waits on
// its first phase, which nothing completes.  The bounded wait gives up after
// the context's budget and records DEV_WAIT_TIMEOUT; no copy is in flight and
// no other thread depends on the barrier, so the CTA simply returns.
__global__ void k_wait_selftest(int* err) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_fence_init();
    mbar_wait_bounded(&bar, 0, err);
  }
}

void launch_wait_selftest(int* err, cudaStream_t st) {
  count_launch();
  k_wait_selftest<<<1, 32, 0, st>>>(err);
}

// ============================================================================
// J
// ============================================================================
// W[s*ldB + k]: the density folded onto the stored tile elements so that
// w_P = sum_k B[P,k] W[k] reproduces REST's per-P scalar:
//   mode 0 (full dot, scf_io/mod.rs:2451-2457): off-diagonal tiles carry
//          D[mu,nu] + D[nu,mu], diagonal tiles D[mu,nu] (both triangles stored);
//   mode 1 (packed formula, :2513-2527): off-diagonal tiles 2 D[mu,nu] (mu < nu),
//          diagonal tiles D[min, max], which sums to 2 sum_{mu<=nu} - sum_diag.
__global__ void __launch_bounds__(256) k_j_weights(int64_t n, int64_t ldB, const double* __restrict__ dm, int nspin,
                                                   int mode, double* __restrict__ W, int* err) {
  const int64_t total = (int64_t)nspin * ldB;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = e / ldB, k = e - s * ldB;
    const int64_t t = k >> 10;
    const int rc = (int)(k & 1023), r = rc & 31, c = rc >> 5;
    const int64_t J = tri_root(t), I = t - J * (J + 1) / 2;
    const int64_t mu = I * TS + r, nu = J * TS + c;
    double v = 0.0;
    if (mu < n && nu < n) {
      const double* D = dm + s * n * n;
      if (I < J) {
        v = mode == 0 ? D[mu + n * nu] + D[nu + n * mu] : 2.0 * D[mu + n * nu];
      } else {
        const int64_t i = mu < nu ? mu : nu, j = mu < nu ? nu : mu;
        v = mode == 0 ? D[mu + n * nu] : D[i + n * j];
      }
      flag_nonfinite(err, v);
    }
    W[e] = v;
  }
}

void launch_j_weights(const Geom& g, const double* dm, int nspin, int mode, double* W, int* err, cudaStream_t st) {
  const int64_t total = nspin * g.ldB;
  const unsigned blocks = (unsigned)std::min<int64_t>(cdiv(total, 256), 148 * 16);
  count_launch();
  k_j_weights<<<blocks, 256, 0, st>>>(g.n, g.ldB, dm, nspin, mode, W, err);
}

__device__ __forceinline__ double2 ld_stream(const double2* p) { return __ldcs(p); }

template <int NS>
__device__ __forceinline__ void block_reduce_store(double (&s)[NS], double* out, int64_t stride) {
  __shared__ double red[NS][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int i = 0; i < NS; ++i)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < NS; ++i) red[i][warp] = s[i];
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      double t = 0.0;
      for (int w = 0; w < nw; ++w) t += red[i][w];
      out[i * stride] = t;
    }
  }
}

// Pass 1: one CTA per aux row P; the row streams once from HBM (evict-first),
// the weights stay in L2.  Fixed summation order: deterministic.
template <int NS>
__global__ void __launch_bounds__(256) k_j_pass1(const double* __restrict__ B, const double* __restrict__ W,
                                                 int64_t ldB, int64_t naux, double* __restrict__ w) {
  const int64_t P = blockIdx.x;
  const double2* b = reinterpret_cast<const double2*>(B + P * ldB);
  const double2* w0 = reinterpret_cast<const double2*>(W);
  const double2* w1 = reinterpret_cast<const double2*>(W + ldB);
  const int64_t nq = ldB / 2;
  double s[NS];
  double s2[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) s[i] = s2[i] = 0.0;
  int64_t q = threadIdx.x;
  constexpr int U = 4;
  for (; q + (U - 1) * 256 < nq; q += U * 256) {
    double2 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = ld_stream(b + q + u * 256);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double2 a = __ldg(w0 + q + u * 256);
      s[0] = fma(x[u].x, a.x, s[0]);
      s2[0] = fma(x[u].y, a.y, s2[0]);
      if (NS == 2) {
        const double2 c = __ldg(w1 + q + u * 256);
        s[NS - 1] = fma(x[u].x, c.x, s[NS - 1]);
        s2[NS - 1] = fma(x[u].y, c.y, s2[NS - 1]);
      }
    }
  }
  for (; q < nq; q += 256) {
    const double2 xv = ld_stream(b + q);
    const double2 a = __ldg(w0 + q);
    s[0] = fma(xv.x, a.x, s[0]);
    s2[0] = fma(xv.y, a.y, s2[0]);
    if (NS == 2) {
      const double2 c = __ldg(w1 + q);
      s[NS - 1] = fma(xv.x, c.x, s[NS - 1]);
      s2[NS - 1] = fma(xv.y, c.y, s2[NS - 1]);
    }
  }
#pragma unroll
  for (int i = 0; i < NS; ++i) s[i] += s2[i];
  block_reduce_store<NS>(s, w + P, naux);
}

void launch_j_pass1(const Geom& g, const double* B, const double* W, int nspin, double* w, cudaStream_t st) {
  count_launch();
  if (nspin == 2)
    k_j_pass1<2><<<(unsigned)g.naux, 256, 0, st>>>(B, W, g.ldB, g.naux, w);
  else
    k_j_pass1<1><<<(unsigned)g.naux, 256, 0, st>>>(B, W, g.ldB, g.naux, w);
}

int j_pass2_splits(const Geom& g) {
  const int64_t threads_per_split = g.ldB / 2;
  const int64_t target = 148LL * 2048 * 2;
  int64_t s = cdiv(target, threads_per_split);
  s = std::max<int64_t>(1, std::min<int64_t>(s, std::min<int64_t>(g.naux, 64)));
  return (int)s;
}

// Pass 2: each thread owns two adjacent stored elements (16 bytes) and walks
// the aux rows of its split; warps read 512 contiguous bytes per row.
template <int NS>
__global__ void __launch_bounds__(256) k_j_pass2(const double* __restrict__ B, const double* __restrict__ w,
                                                 int64_t ldB, int64_t naux, int splits, double* __restrict__ Jpart) {
  const int64_t nq = ldB / 2;
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int sp = blockIdx.y;
  const int64_t p0 = naux * sp / splits, p1 = naux * (sp + 1) / splits;
  if (q >= nq) return;
  const double2* b = reinterpret_cast<const double2*>(B) + q;
  double2 a[NS];
#pragma unroll
  for (int i = 0; i < NS; ++i) a[i] = make_double2(0.0, 0.0);
  int64_t p = p0;
  constexpr int U = 4;
  for (; p + U - 1 < p1; p += U) {
    double2 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = ld_stream(b + (p + u) * nq);
#pragma unroll
    for (int u = 0; u < U; ++u) {
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        const double wp = __ldg(w + i * naux + p + u);
        a[i].x = fma(x[u].x, wp, a[i].x);
        a[i].y = fma(x[u].y, wp, a[i].y);
      }
    }
  }
  for (; p < p1; ++p) {
    const double2 xv = ld_stream(b + p * nq);
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      const double wp = __ldg(w + i * naux + p);
      a[i].x = fma(xv.x, wp, a[i].x);
      a[i].y = fma(xv.y, wp, a[i].y);
    }
  }
#pragma unroll
  for (int i = 0; i < NS; ++i) reinterpret_cast<double2*>(Jpart + ((int64_t)sp * NS + i) * ldB)[q] = a[i];
}

void launch_j_pass2(const Geom& g, const double* B, const double* w, int nspin, int splits, double* Jpart,
                    cudaStream_t st) {
  dim3 grid((unsigned)cdiv(g.ldB / 2, 256), (unsigned)splits);
  count_launch();
  if (nspin == 2)
    k_j_pass2<2><<<grid, 256, 0, st>>>(B, w, g.ldB, g.naux, splits, Jpart);
  else
    k_j_pass2<1><<<grid, 256, 0, st>>>(B, w, g.ldB, g.naux, splits, Jpart);
}

__global__ void __launch_bounds__(256) k_j_finalize(int64_t n, int64_t npair, int64_t ldB,
                                                    const double* __restrict__ Jpart, int nspin, int splits,
                                                    double scale, int out_kind, double* __restrict__ out) {
  const int64_t per = out_kind == 0 ? npair : n * n;
  const int64_t total = nspin * per;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = e / per, t = e - s * per;
    int64_t i, j;
    if (out_kind == 0) {
      j = tri_root(t);
      i = t - j * (j + 1) / 2;
    } else {
      const int64_t mu = t % n, nu = t / n;
      i = mu < nu ? mu : nu;
      j = mu < nu ? nu : mu;
    }
    const int64_t k = tile_pair_index(i / TS, j / TS) * TILE_ELEMS + (i % TS) + TS * (j % TS);
    double v = 0.0;
    for (int sp = 0; sp < splits; ++sp) v += Jpart[((int64_t)sp * nspin + s) * ldB + k];
    out[e] = v * scale;
  }
}

// Sum over the splits of part(sp) for 32 consecutive elements per CTA: eight
// groups of threads take the splits in turn, and their sums are added in order.
// With many splits (few elements) one thread per element waits for its loads one
// after another: J's and K's sums took 28 and 20 of the 85 us that a 24-function
// molecule's kernels take, and its whole build took 124 us, 99 with this form.
constexpr int WIDE_SPLITS = 8;  // from one split per group on; below, groups would idle
template <class Part>
__device__ __forceinline__ double wide_sum(int splits, bool in, const Part& part) {
  __shared__ double red[8][32];
  double v = 0.0;
  if (in)
#pragma unroll 4
    for (int sp = threadIdx.y; sp < splits; sp += 8) v += part(sp);
  red[threadIdx.y][threadIdx.x] = v;
  __syncthreads();
  v = 0.0;
#pragma unroll
  for (int y = 0; y < 8; ++y) v += red[y][threadIdx.x];
  return v;
}

__global__ void __launch_bounds__(256) k_j_finalize_wide(int64_t n, int64_t npair, int64_t ldB,
                                                         const double* __restrict__ Jpart, int nspin, int splits,
                                                         double scale, int out_kind, double* __restrict__ out) {
  const int64_t per = out_kind == 0 ? npair : n * n;
  const int64_t e = (int64_t)blockIdx.x * 32 + threadIdx.x;
  const bool in = e < nspin * per;
  int64_t s = 0, k = 0;
  if (in) {
    s = e / per;
    const int64_t t = e - s * per;
    int64_t i, j;
    if (out_kind == 0) {
      j = tri_root(t);
      i = t - j * (j + 1) / 2;
    } else {
      const int64_t mu = t % n, nu = t / n;
      i = mu < nu ? mu : nu;
      j = mu < nu ? nu : mu;
    }
    k = tile_pair_index(i / TS, j / TS) * TILE_ELEMS + (i % TS) + TS * (j % TS);
  }
  const double v = wide_sum(splits, in, [&](int sp) { return Jpart[((int64_t)sp * nspin + s) * ldB + k]; });
  if (in && threadIdx.y == 0) out[e] = v * scale;
}

void launch_j_finalize(const Geom& g, const double* Jpart, int nspin, int splits, double scale, int out_kind,
                       double* out, cudaStream_t st) {
  const int64_t total = nspin * (out_kind == 0 ? g.npair : g.n * g.n);
  if (splits >= WIDE_SPLITS) {
    count_launch();
    k_j_finalize_wide<<<(unsigned)cdiv(total, 32), dim3(32, 8), 0, st>>>(g.n, g.npair, g.ldB, Jpart, nspin, splits,
                                                                         scale, out_kind, out);
    return;
  }
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(total, 256), 148 * 16));
  count_launch();
  k_j_finalize<<<blocks, 256, 0, st>>>(g.n, g.npair, g.ldB, Jpart, nspin, splits, scale, out_kind, out);
}

// ============================================================================
// K
// ============================================================================
// Right operand of the half-transform: the occupied columns of each spin,
// scaled by sqrt(occupation), so that (B_P Cw)(B_P Cw)^T = B_P C occ C^T B_P
// (REST forms Y = X diag(occ) and Y X^T, scf_io/mod.rs:2797-2803).  Spin s
// occupies columns [coff_s, coff_s + nw_s) with coff_1 = round_up(nw_0, 32).
__global__ void __launch_bounds__(256) k_prepare_c(int64_t n, const double* __restrict__ eigv, int64_t ld_eigv,
                                                   int64_t stride_eigv, const double* __restrict__ occ,
                                                   int64_t stride_occ, int64_t nw0, int64_t nw1, int64_t coff1,
                                                   int nspin, int64_t ldc, int64_t ocols, double* __restrict__ Cw,
                                                   int* err) {
  const int64_t total = ldc * ocols;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = e % ldc, col = e / ldc;
    double v = 0.0;
    int s = -1;
    int64_t i = 0;
    if (col < nw0) {
      s = 0;
      i = col;
    } else if (nspin == 2 && col >= coff1 && col < coff1 + nw1) {
      s = 1;
      i = col - coff1;
    }
    if (s >= 0 && row < n) {
      const double o = occ[s * stride_occ + i];
      v = eigv[s * stride_eigv + row + ld_eigv * i] * sqrt(o);
      flag_nonfinite(err, v);  // NaN/Inf orbitals or occupations (and negative occupations)
    }
    Cw[e] = v;
  }
}

void launch_k_prepare_c(const Geom& g, const double* eigv, int64_t ld_eigv, int64_t stride_eigv, const double* occ,
                        int64_t stride_occ, const int64_t* nw, int nspin, int64_t ldc, int64_t ocols, double* Cw,
                        int* err, cudaStream_t st) {
  const int64_t coff1 = round_up(nw[0], TS);
  const int64_t total = ldc * ocols;
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(total, 256), 148 * 16));
  count_launch();
  k_prepare_c<<<blocks, 256, 0, st>>>(g.n, eigv, ld_eigv, stride_eigv, occ, stride_occ, nw[0], nspin == 2 ? nw[1] : 0,
                                      coff1, nspin, ldc, ocols, Cw, err);
}

__global__ void __launch_bounds__(256) k_pad_square(const double* __restrict__ src, int64_t n, int64_t ldsrc,
                                                    int64_t ldc, double* __restrict__ dst, int* err) {
  const int64_t total = ldc * ldc;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e % ldc, c = e / ldc;
    double v = 0.0;
    if (r < n && c < n) {
      v = src[r + ldsrc * c];
      flag_nonfinite(err, v);
    }
    dst[e] = v;
  }
}

void launch_pad_square(const double* src, int64_t n, int64_t ldsrc, int64_t ldc, double* dst, int* err,
                       cudaStream_t st) {
  const int64_t total = ldc * ldc;
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(total, 256), 148 * 16));
  count_launch();
  k_pad_square<<<blocks, 256, 0, st>>>(src, n, ldsrc, ldc, dst, err);
}

// ---- half-transform: X_p = B_p W ------------------------------------------
// CTA shapes (selected per context; rows x cols, compute warps, stages, staging):
using HtCfg0 = DmmaCfg<2, 2, 2, 2, 3, true>;  // 64 x 64, 4 warps of 32 x 32, cp.async, 3 stages (2 CTAs/SM)
using HtCfg1 = DmmaCfg<2, 2, 2, 2, 2, true>;  // 64 x 64, cp.async, 2 stages (3 CTAs/SM)
using HtCfg2 = DmmaCfg<2, 2, 2, 2, 4, true>;  // 64 x 64, cp.async, 4 stages (1 CTA/SM)
using HtCfg3 = DmmaCfg<2, 2, 2, 2, 3>;        // 64 x 64, bulk copies + producer warp, 3 stages
using HtCfg4 = DmmaCfg<4, 2, 4, 2, 2, true>;  // 128 x 64, 8 warps of 32 x 32, cp.async, 2 stages (2 CTAs/SM)
using HtCfg5 = DmmaCfg<2, 4, 2, 2, 2, true>;  // 64 x 128, 4 warps of 32 x 64, cp.async, 2 stages (2 CTAs/SM)

// Register budget: two CTAs per SM for the 256-thread shape (128 registers) and
// for the shape with 32 x 64 warp tiles (up to 255 registers).
template <class Cfg>
constexpr int min_ctas() {
  // 4-warp 64x64 shapes whose shared memory lets three CTAs share an SM ask
  // for registers that let them (<= 170 per thread)
  if (Cfg::THREADS == 128 && Cfg::FM * Cfg::FN == 16 && 3 * Cfg::SMEM_BYTES <= 227 * 1024) return 3;
  return (Cfg::THREADS >= 256 || Cfg::FM * Cfg::FN >= 32) ? 2 : 1;
}

struct HalfTransformSched {
  const double* Bp;  // row P of the tile-packed tensor
  const double* W;
  int64_t ldw;
  int nt, I0, col0;
  int xcol0;  // first remainder column (CTAs of the last full column block)
  __device__ SlotSrc a(int kt, int mt) const {
    const int I = I0 + mt, J = kt;
    if (I >= nt) return {nullptr, TS, 0};
    if (I <= J) return {Bp + tile_pair_index(I, J) * TILE_ELEMS, TS, 0};
    return {Bp + tile_pair_index(J, I) * TILE_ELEMS, TS, 1};
  }
  __device__ SlotSrc b(int kt, int ntl) const {
    return {W + (int64_t)kt * TS + (int64_t)(col0 + ntl * TS) * ldw, ldw, 0};
  }
  __device__ SlotSrc x(int kt) const { return {W + (int64_t)kt * TS + (int64_t)xcol0 * ldw, ldw, 0}; }
};

// Only the rows of the last k tile below n can be non-zero.
struct LastTileK {
  int last, lastk;
  __device__ int operator()(int kt) const { return kt == last ? lastk : TS; }
};

// Grid: blockIdx.x = cb + ncb * (rb + nrb * p), so that the column blocks of
// one row block run back to back and share its B tiles in L2.
// XF > 0: the CTAs of the last column block (cb == ncb - 1) also compute the
// XF * 8 remainder columns from xcol0 on (see ExtraCols).
// wpart != nullptr: also J's scalars.  Consumer warp k of CTA bid writes its
// share of w_P,s = <W_s, X_P,s> = sum over its outputs of X_P[m, c] W[m, c]
// (W = C scaled by sqrt(occ), zero padded, so w_P,s = B_P : D_s with
// D_s = W_s W_s^T) to wpart[2 (bid CWARPS + k) + s]; s = 0 for the columns
// below coff1, else 1.
template <class Cfg, int XF = 0>
__global__ void __launch_bounds__(Cfg::THREADS, min_ctas<Cfg>()) k_half_transform(const double* __restrict__ B, int64_t ldB, int64_t p0,
                                                                 int nrb, int ncb, const double* __restrict__ W,
                                                                 int64_t ldw, int n, int nt, int ncol_valid,
                                                                 double* __restrict__ X, int64_t ldx, XMap xm,
                                                                 int* err, int xcol0, double* __restrict__ wpart,
                                                                 int coff1) {
  extern __shared__ __align__(128) double smem[];
  const int64_t bid = blockIdx.x;
  const int cb = (int)(bid % ncb);
  const int64_t rest = bid / ncb;
  const int64_t pl = rest / nrb;
  const int I0 = (int)(rest % nrb) * Cfg::MT;
  const int col0 = cb * Cfg::BN;
  if (I0 * TS >= n || col0 >= ncol_valid) {  // padding only, which nothing reads
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (wpart && lane < 2 && warp < Cfg::CWARPS) wpart[2 * (bid * Cfg::CWARPS + warp) + lane] = 0.0;
    return;
  }
  HalfTransformSched sc{B + (p0 + pl) * ldB, W, ldw, nt, I0, col0, xcol0};
  double acc[Cfg::FM][Cfg::FN][2];
  ExtraCols<XF> xc;
  xc.on = XF > 0 && cb == ncb - 1;
  const LastTileK kv{nt - 1, n - (nt - 1) * TS};
  if (!dmma_mainloop<Cfg, HalfTransformSched, LastTileK, XF>(sc, nt, smem, acc, err, n - I0 * TS,
                                                             ncol_valid - col0, kv, &xc))
    return;
  double* Xr = X + (int64_t)I0 * TS;
  dmma_for_each<Cfg>(acc, [&](int m, int c, double v0, double v1) {
    const int64_t d0 = xm.dst(pl, col0 + c), d1 = xm.dst(pl, col0 + c + 1);
    if (d0 >= 0) Xr[m + d0 * ldx] = v0;
    if (d1 >= 0) Xr[m + d1 * ldx] = v1;
  });
  if constexpr (XF > 0) {
    if (xc.on) {
      const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      const int wm = warp / Cfg::WN, wn = warp % Cfg::WN;
#pragma unroll
      for (int e = 0; e < 2; ++e)
#pragma unroll
        for (int j = 0; j < XF; ++j) {
          const int m = wm * Cfg::WTM + (wn * 2 + e) * 8 + (lane >> 2);
          const int c = xcol0 + 8 * j + 2 * (lane & 3);
          const int64_t d0 = c < ncol_valid ? xm.dst(pl, c) : -1, d1 = c + 1 < ncol_valid ? xm.dst(pl, c + 1) : -1;
          if (d0 >= 0) Xr[m + d0 * ldx] = xc.acc[e][j][0];
          if (d1 >= 0) Xr[m + d1 * ldx] = xc.acc[e][j][1];
        }
    }
  }
  if (wpart) {
    // this warp's share of <W, X_P> per spin
    double s0 = 0.0, s1 = 0.0;
    const double* Wr = W + (int64_t)I0 * TS;
    dmma_for_each<Cfg>(acc, [&](int m, int c, double v0, double v1) {
      const int c0 = col0 + c;
      const double t0 = v0 * Wr[m + (int64_t)c0 * ldw], t1 = v1 * Wr[m + (int64_t)(c0 + 1) * ldw];
      if (c0 < coff1) s0 += t0; else s1 += t0;
      if (c0 + 1 < coff1) s0 += t1; else s1 += t1;
    });
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if constexpr (XF > 0) {
      if (xc.on) {
        const int wm = warp / Cfg::WN, wn = warp % Cfg::WN;
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int j = 0; j < XF; ++j) {
            const int m = wm * Cfg::WTM + (wn * 2 + e) * 8 + (lane >> 2);
            const int c = xcol0 + 8 * j + 2 * (lane & 3);
            const double t0 = xc.acc[e][j][0] * Wr[m + (int64_t)c * ldw];
            const double t1 = xc.acc[e][j][1] * Wr[m + (int64_t)(c + 1) * ldw];
            if (c < coff1) s0 += t0; else s1 += t0;
            if (c + 1 < coff1) s0 += t1; else s1 += t1;
          }
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s0 += __shfl_xor_sync(0xffffffffu, s0, o);
      s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    }
    if (lane == 0) {
      wpart[2 * (bid * Cfg::CWARPS + warp)] = s0;
      wpart[2 * (bid * Cfg::CWARPS + warp) + 1] = s1;
    }
  }
}

// w[s][p0 + p] = the sum, in a fixed order, of the per_row warp shares of aux
// row p (one warp per row).
__global__ void __launch_bounds__(256) k_j_wreduce(const double* __restrict__ wpart, int64_t np, int per_row,
                                                   int nspin, int64_t naux, int64_t p0, double* __restrict__ w) {
  const int lane = threadIdx.x & 31;
  for (int64_t pl = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; pl < np;
       pl += ((int64_t)gridDim.x * blockDim.x) >> 5) {
    const double* src = wpart + pl * per_row * 2;
    double a = 0.0, b = 0.0;
    for (int t = lane; t < per_row; t += 32) {
      a += src[2 * t];
      b += src[2 * t + 1];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      b += __shfl_xor_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
      w[p0 + pl] = a;
      if (nspin == 2) w[naux + p0 + pl] = b;
    }
  }
}

void launch_j_wreduce(const double* wpart, int64_t np, int per_row, int nspin, int64_t naux, int64_t p0, double* w,
                      cudaStream_t st) {
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(np, 8), 148 * 8));
  count_launch();
  k_j_wreduce<<<blocks, 256, 0, st>>>(wpart, np, per_row, nspin, naux, p0, w);
}

// J scalars requested by the caller of launch_half_transform (see JFuse).
struct JFuse {
  double* wpart;  // scratch, 2 doubles per CTA
  double* w;      // [spin][naux]
  int nspin, coff1;
  int64_t naux;
};

template <class Cfg, int XF = 0>
static void half_transform_launch(const Geom& g, const double* B, int64_t p0, int64_t np, const double* W,
                                  int64_t ldw, int ncb, int64_t ncol_valid, double* X, int64_t ldx, const XMap& xm,
                                  int* err, int xcol0, const JFuse* jf, cudaStream_t st) {
  cudaFuncSetAttribute(k_half_transform<Cfg, XF>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)Cfg::SMEM_BYTES);
  const int nrb = (int)(ldx / Cfg::BM);
  double* wpart = jf ? jf->wpart : nullptr;
  count_launch();
  k_half_transform<Cfg, XF><<<(unsigned)(np * nrb * ncb), Cfg::THREADS, Cfg::SMEM_BYTES, st>>>(
      B, g.ldB, p0, nrb, ncb, W, ldw, (int)g.n, (int)g.nt, (int)ncol_valid, X, ldx, xm, err, xcol0, wpart,
      jf ? jf->coff1 : 1 << 30);
  if (wpart) launch_j_wreduce(wpart, np, nrb * ncb * Cfg::CWARPS, jf->nspin, jf->naux, p0, jf->w, st);
}

template <class Cfg>
static void half_transform_cfg(const Geom& g, const double* B, int64_t p0, int64_t np, const double* W, int64_t ldw,
                               int64_t ncol, int64_t ncol_valid, double* X, int64_t ldx, const XMap& xm, int* err,
                               const JFuse* jf, cudaStream_t st) {
  half_transform_launch<Cfg>(g, B, p0, np, W, ldw, (int)(ncol / Cfg::BN), ncol_valid, X, ldx, xm, err, 0, jf, st);
}

// The default shape: when the valid columns end at most 16 past a multiple of
// 64, the last full column block also computes those remainder columns (one or
// two extra fragments) instead of a block of CTAs for them alone.
template <>
void half_transform_cfg<HtCfg1>(const Geom& g, const double* B, int64_t p0, int64_t np, const double* W,
                                int64_t ldw, int64_t ncol, int64_t ncol_valid, double* X, int64_t ldx,
                                const XMap& xm, int* err, const JFuse* jf, cudaStream_t st) {
  const int64_t full = ncol_valid / HtCfg1::BN, rem = ncol_valid - full * HtCfg1::BN;
  const int xcol0 = (int)(full * HtCfg1::BN);
  if (full >= 1 && rem > 0 && rem <= 8)
    return half_transform_launch<HtCfg1, 1>(g, B, p0, np, W, ldw, (int)full, ncol_valid, X, ldx, xm, err, xcol0,
                                            jf, st);
  if (full >= 1 && rem > 8 && rem <= 16)
    return half_transform_launch<HtCfg1, 2>(g, B, p0, np, W, ldw, (int)full, ncol_valid, X, ldx, xm, err, xcol0,
                                            jf, st);
  half_transform_launch<HtCfg1>(g, B, p0, np, W, ldw, (int)(ncol / HtCfg1::BN), ncol_valid, X, ldx, xm, err, 0, jf,
                                st);
}

int64_t half_transform_warps(const Geom& g, int64_t np, int64_t ldx, int64_t ncol) {
  switch (g.ht_cfg) {
    case 1: return np * (ldx / HtCfg1::BM) * (ncol / HtCfg1::BN) * HtCfg1::CWARPS;
    case 2: return np * (ldx / HtCfg2::BM) * (ncol / HtCfg2::BN) * HtCfg2::CWARPS;
    case 3: return np * (ldx / HtCfg3::BM) * (ncol / HtCfg3::BN) * HtCfg3::CWARPS;
    case 4: return np * (ldx / HtCfg4::BM) * (ncol / HtCfg4::BN) * HtCfg4::CWARPS;
    case 5: return np * (ldx / HtCfg5::BM) * (ncol / HtCfg5::BN) * HtCfg5::CWARPS;
    default: return np * (ldx / HtCfg0::BM) * (ncol / HtCfg0::BN) * HtCfg0::CWARPS;
  }
}

void launch_half_transform(const Geom& g, const double* B, int64_t p0, int64_t np, const double* W, int64_t ldw,
                           int64_t ncol, int64_t ncol_valid, double* X, int64_t ldx, const XMap& xm, int* err,
                           cudaStream_t st, double* wpart, double* w, int nspin, int coff1) {
  JFuse jfs{wpart, w, nspin, coff1, g.naux};
  const JFuse* jf = wpart ? &jfs : nullptr;
  switch (g.ht_cfg) {
    case 1: return half_transform_cfg<HtCfg1>(g, B, p0, np, W, ldw, ncol, ncol_valid, X, ldx, xm, err, jf, st);
    case 2: return half_transform_cfg<HtCfg2>(g, B, p0, np, W, ldw, ncol, ncol_valid, X, ldx, xm, err, jf, st);
    case 3: return half_transform_cfg<HtCfg3>(g, B, p0, np, W, ldw, ncol, ncol_valid, X, ldx, xm, err, jf, st);
    case 4: return half_transform_cfg<HtCfg4>(g, B, p0, np, W, ldw, ncol, ncol_valid, X, ldx, xm, err, jf, st);
    case 5: return half_transform_cfg<HtCfg5>(g, B, p0, np, W, ldw, ncol, ncol_valid, X, ldx, xm, err, jf, st);
    default: return half_transform_cfg<HtCfg0>(g, B, p0, np, W, ldw, ncol, ncol_valid, X, ldx, xm, err, jf, st);
  }
}

// ---- rank update: Kpart = sum_p X_p X_p^T ------------------------------------
// K is accumulated in 128 x 128 blocks; a CTA computes one (BM x BN) sub-block
// of one block.  CTA shapes (selected per context):
using RkCfg0 = DmmaCfg<2, 2, 2, 2, 3, true>;  // 64 x 64, 4 warps of 32 x 32, cp.async, 3 stages (2 CTAs/SM)
using RkCfg1 = DmmaCfg<2, 2, 2, 2, 2, true>;  // 64 x 64, cp.async, 2 stages (3 CTAs/SM)
using RkCfg2 = DmmaCfg<2, 2, 2, 2, 4, true>;  // 64 x 64, cp.async, 4 stages (1 CTA/SM)
using RkCfg3 = DmmaCfg<2, 2, 2, 2, 3>;        // 64 x 64, bulk copies + producer warp, 3 stages
using RkCfg4 = DmmaCfg<4, 2, 4, 2, 2, true>;  // 128 x 64, 8 warps, cp.async, 2 stages (2 CTAs/SM)
using RkCfg5 = DmmaCfg<2, 4, 2, 2, 2, true>;  // 64 x 128, 4 warps of 32 x 64, cp.async, 2 stages (2 CTAs/SM)
constexpr int KB = 128;                       // K block edge

static int rk_subs(int cfg) { return cfg >= 4 ? 2 : 4; }  // CTA sub-blocks of a 128 x 128 K block
static int rk_ctas_per_sm(int cfg) { return cfg == 1 ? 3 : cfg == 2 ? 1 : 2; }

int64_t k_block_pairs(const Geom& g, int full) {
  const int64_t nkb = cdiv(g.n, KB);
  return full ? nkb * nkb : nkb * (nkb + 1) / 2;
}

__device__ __forceinline__ void block_pair(int64_t q, int full, int64_t nkb, int64_t& Ib, int64_t& Jb) {
  if (full) {
    Ib = q % nkb;
    Jb = q / nkb;
  } else {
    Jb = tri_root(q);
    Ib = q - Jb * (Jb + 1) / 2;
  }
}

int k_rank_splits(const Geom& g, int64_t np, int full) {
  const int64_t ctas = k_block_pairs(g, full) * rk_subs(g.rk_cfg);
  int64_t s = cdiv(2 * 148 * rk_ctas_per_sm(g.rk_cfg), ctas);
  s = std::max<int64_t>(1, std::min<int64_t>(s, np));
  return (int)s;
}

// Sub-block (hm, hn) of block pair q for CTA tile BM x BN; false when the
// sub-block lies strictly below the diagonal of a diagonal block (never read).
template <class Cfg>
__device__ __forceinline__ bool sub_block(int64_t bq, int full, int64_t nkb, int64_t& q, int64_t& row0,
                                          int64_t& col0, int64_t& off) {
  constexpr int SM = KB / Cfg::BM, SN = KB / Cfg::BN;
  q = bq / (SM * SN);
  const int sub = (int)(bq % (SM * SN));
  const int hm = sub % SM, hn = sub / SM;
  int64_t Ib, Jb;
  block_pair(q, full, nkb, Ib, Jb);
  row0 = Ib * KB + hm * Cfg::BM;
  col0 = Jb * KB + hn * Cfg::BN;
  off = hm * Cfg::BM + (int64_t)KB * (hn * Cfg::BN);
  return full || Ib != Jb || hm * Cfg::BM < (hn + 1) * Cfg::BN;
}

// Operands of the rank update: this spin's half-transformed orbitals as one
// matrix with column k = p * nw + i (aux row p of the chunk, orbital i), so the
// contraction runs over k without padding between aux rows.
struct RankSched {
  const double* X;
  int64_t ldx, k0;
  int64_t mrow0, nrow0;
  __device__ SlotSrc a(int kt, int mt) const {
    return {X + mrow0 + mt * TS + (k0 + (int64_t)kt * TS) * ldx, ldx, 0};
  }
  __device__ SlotSrc b(int kt, int ntl) const {
    return {X + nrow0 + ntl * TS + (k0 + (int64_t)kt * TS) * ldx, ldx, 1};
  }
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, min_ctas<Cfg>()) k_rank_update(const double* __restrict__ X, int64_t ldx,
                                                              int64_t np, int nw, int n, int splits, int full,
                                                              int64_t nkb, int64_t pairs, double* __restrict__ Kpart,
                                                              int* err) {
  extern __shared__ __align__(128) double smem[];
  const int sp = blockIdx.y;
  int64_t q, row0, col0, off;
  if (!sub_block<Cfg>(blockIdx.x, full, nkb, q, row0, col0, off) || row0 >= n || col0 >= n) return;
  const int64_t pa = np * sp / splits, pb = np * (sp + 1) / splits;
  const int64_t kcount = (pb - pa) * nw;
  RankSched sc{X, ldx, pa * nw, row0, col0};
  double acc[Cfg::FM][Cfg::FN][2];
  const int ktiles = (int)((kcount + TS - 1) / TS);
  const LastTileK kv{ktiles - 1, (int)(kcount - (int64_t)(ktiles - 1) * TS)};
  if (!dmma_mainloop<Cfg>(sc, ktiles, smem, acc, err, n - (int)row0, n - (int)col0, kv)) return;
  double* out = Kpart + ((int64_t)sp * pairs + q) * (KB * KB) + off;
  dmma_for_each<Cfg>(acc, [&](int m, int c, double v0, double v1) {
    out[m + KB * c] = v0;
    out[m + KB * (c + 1)] = v1;
  });
}

template <class Cfg>
static void rank_update_cfg(const Geom& g, const double* X, int64_t ldx, int64_t np, int64_t nw, int splits, int full,
                            double* Kpart, int* err, cudaStream_t st) {
  cudaFuncSetAttribute(k_rank_update<Cfg>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM_BYTES);
  const int64_t nkb = cdiv(g.n, KB);
  const int64_t pairs = k_block_pairs(g, full);
  constexpr int subs = (KB / Cfg::BM) * (KB / Cfg::BN);
  dim3 grid((unsigned)(pairs * subs), (unsigned)splits);
  count_launch();
  k_rank_update<Cfg><<<grid, Cfg::THREADS, Cfg::SMEM_BYTES, st>>>(X, ldx, np, (int)nw, (int)g.n, splits, full, nkb,
                                                                   pairs, Kpart, err);
}

void launch_k_rank_update(const Geom& g, const double* X, int64_t ldx, int64_t np, int64_t nw, int splits, int full,
                          double* Kpart, int* err, cudaStream_t st) {
  switch (g.rk_cfg) {
    case 1: return rank_update_cfg<RkCfg1>(g, X, ldx, np, nw, splits, full, Kpart, err, st);
    case 2: return rank_update_cfg<RkCfg2>(g, X, ldx, np, nw, splits, full, Kpart, err, st);
    case 3: return rank_update_cfg<RkCfg3>(g, X, ldx, np, nw, splits, full, Kpart, err, st);
    case 4: return rank_update_cfg<RkCfg4>(g, X, ldx, np, nw, splits, full, Kpart, err, st);
    case 5: return rank_update_cfg<RkCfg5>(g, X, ldx, np, nw, splits, full, Kpart, err, st);
    default: return rank_update_cfg<RkCfg0>(g, X, ldx, np, nw, splits, full, Kpart, err, st);
  }
}

// ---- dm form: Kpart = sum_p T_p B_p ------------------------------------------
struct KdmSched {
  const double* T;
  int64_t ldt, stp;
  const double* B;
  int64_t ldB;
  int64_t pg0;  // global aux index of local p = 0
  int64_t p0;   // first local p of this split
  int nt;
  int64_t mrow0;
  int nb0;  // first nu tile of this CTA
  __device__ SlotSrc a(int kt, int mt) const {
    const int64_t p = p0 + kt / nt;
    const int kb = kt % nt;
    return {T + p * stp + mrow0 + mt * TS + (int64_t)kb * TS * ldt, ldt, 0};
  }
  __device__ SlotSrc b(int kt, int ntl) const {
    const int64_t p = p0 + kt / nt;
    const int kb = kt % nt;
    const int nb = nb0 + ntl;
    if (nb >= nt) return {nullptr, TS, 0};
    const double* Bp = B + (pg0 + p) * ldB;
    if (kb <= nb) return {Bp + tile_pair_index(kb, nb) * TILE_ELEMS, TS, 0};
    return {Bp + tile_pair_index(nb, kb) * TILE_ELEMS, TS, 1};
  }
};

// Valid k columns of the last tile of every aux row (k tiles run row by row,
// ctiles per row).
struct RankK {
  int ctiles, lastk;
  __device__ int operator()(int kt) const { return (kt % ctiles) == ctiles - 1 ? lastk : TS; }
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, min_ctas<Cfg>()) k_dm_update(const double* __restrict__ T, int64_t ldt, int64_t stp,
                                                            const double* __restrict__ B, int64_t ldB, int64_t pg0,
                                                            int64_t np, int n, int nt, int splits, int full,
                                                            int64_t nkb, int64_t pairs, double* __restrict__ Kpart,
                                                            int* err) {
  extern __shared__ __align__(128) double smem[];
  const int sp = blockIdx.y;
  int64_t q, row0, col0, off;
  if (!sub_block<Cfg>(blockIdx.x, full, nkb, q, row0, col0, off) || row0 >= n || col0 >= n) return;
  const int64_t pa = np * sp / splits, pb = np * (sp + 1) / splits;
  KdmSched sc{T, ldt, stp, B, ldB, pg0, pa, nt, row0, (int)(col0 / TS)};
  double acc[Cfg::FM][Cfg::FN][2];
  const int ktiles = (int)((pb - pa) * nt);
  if (!dmma_mainloop<Cfg>(sc, ktiles, smem, acc, err, n - (int)row0, n - (int)col0, RankK{nt, n - (nt - 1) * TS}))
    return;
  double* out = Kpart + ((int64_t)sp * pairs + q) * (KB * KB) + off;
  dmma_for_each<Cfg>(acc, [&](int m, int c, double v0, double v1) {
    out[m + KB * c] = v0;
    out[m + KB * (c + 1)] = v1;
  });
}

template <class Cfg>
static void dm_update_cfg(const Geom& g, const double* T, int64_t ldt, int64_t stp, const double* B, int64_t p0,
                          int64_t np, int splits, int full, double* Kpart, int* err, cudaStream_t st) {
  cudaFuncSetAttribute(k_dm_update<Cfg>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM_BYTES);
  const int64_t nkb = cdiv(g.n, KB);
  const int64_t pairs = k_block_pairs(g, full);
  constexpr int subs = (KB / Cfg::BM) * (KB / Cfg::BN);
  dim3 grid((unsigned)(pairs * subs), (unsigned)splits);
  count_launch();
  k_dm_update<Cfg><<<grid, Cfg::THREADS, Cfg::SMEM_BYTES, st>>>(T, ldt, stp, B, g.ldB, p0, np, (int)g.n, (int)g.nt,
                                                                 splits, full, nkb, pairs, Kpart, err);
}

void launch_k_dm_update(const Geom& g, const double* T, int64_t ldt, int64_t stp, const double* B, int64_t p0,
                        int64_t np, int splits, int full, double* Kpart, int* err, cudaStream_t st) {
  switch (g.rk_cfg) {
    case 1: return dm_update_cfg<RkCfg1>(g, T, ldt, stp, B, p0, np, splits, full, Kpart, err, st);
    case 2: return dm_update_cfg<RkCfg2>(g, T, ldt, stp, B, p0, np, splits, full, Kpart, err, st);
    case 3: return dm_update_cfg<RkCfg3>(g, T, ldt, stp, B, p0, np, splits, full, Kpart, err, st);
    case 4: return dm_update_cfg<RkCfg4>(g, T, ldt, stp, B, p0, np, splits, full, Kpart, err, st);
    case 5: return dm_update_cfg<RkCfg5>(g, T, ldt, stp, B, p0, np, splits, full, Kpart, err, st);
    default: return dm_update_cfg<RkCfg0>(g, T, ldt, stp, B, p0, np, splits, full, Kpart, err, st);
  }
}

__global__ void __launch_bounds__(256) k_k_finalize(int64_t n, int64_t npair, const double* __restrict__ Kpart,
                                                    int splits, int full, int64_t nkb, int64_t pairs, double scale,
                                                    int accumulate, int out_kind, double* __restrict__ out) {
  const int64_t total = out_kind == 0 ? npair : n * n;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    int64_t i, j;
    if (out_kind == 0) {
      j = tri_root(e);
      i = e - j * (j + 1) / 2;
    } else {
      i = e % n;
      j = e / n;
    }
    const int64_t Ib = i / KB, Jb = j / KB;
    const int64_t q = full ? Ib + nkb * Jb : Jb * (Jb + 1) / 2 + Ib;
    const int64_t off = (i % KB) + (int64_t)KB * (j % KB);
    double v = 0.0;
    for (int sp = 0; sp < splits; ++sp) v += Kpart[((int64_t)sp * pairs + q) * (KB * KB) + off];
    v *= scale;
    out[e] = accumulate ? out[e] + v : v;
  }
}

__global__ void __launch_bounds__(256) k_k_finalize_wide(int64_t n, int64_t npair, const double* __restrict__ Kpart,
                                                         int splits, int full, int64_t nkb, int64_t pairs,
                                                         double scale, int accumulate, int out_kind,
                                                         double* __restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * 32 + threadIdx.x;
  const bool in = e < (out_kind == 0 ? npair : n * n);
  int64_t at = 0;
  if (in) {
    int64_t i, j;
    if (out_kind == 0) {
      j = tri_root(e);
      i = e - j * (j + 1) / 2;
    } else {
      i = e % n;
      j = e / n;
    }
    const int64_t Ib = i / KB, Jb = j / KB;
    const int64_t q = full ? Ib + nkb * Jb : Jb * (Jb + 1) / 2 + Ib;
    at = q * (KB * KB) + (i % KB) + (int64_t)KB * (j % KB);
  }
  const double v = wide_sum(splits, in, [&](int sp) { return Kpart[(int64_t)sp * pairs * (KB * KB) + at]; }) * scale;
  if (in && threadIdx.y == 0) out[e] = accumulate ? out[e] + v : v;
}

void launch_k_finalize(const Geom& g, const double* Kpart, int splits, int full, double scale, int accumulate,
                       int out_kind, double* out, cudaStream_t st) {
  const int64_t nkb = cdiv(g.n, KB);
  const int64_t pairs = k_block_pairs(g, full);
  const int64_t total = out_kind == 0 ? g.npair : g.n * g.n;
  if (splits >= WIDE_SPLITS) {
    count_launch();
    k_k_finalize_wide<<<(unsigned)cdiv(total, 32), dim3(32, 8), 0, st>>>(g.n, g.npair, Kpart, splits, full, nkb, pairs,
                                                                         scale, accumulate, out_kind, out);
    return;
  }
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(total, 256), 148 * 16));
  count_launch();
  k_k_finalize<<<blocks, 256, 0, st>>>(g.n, g.npair, Kpart, splits, full, nkb, pairs, scale, accumulate, out_kind,
                                       out);
}

// ============================================================================
// Grouped build over a set of molecules (one launch per phase for all of them)
// ============================================================================
// A molecule set's SCFs advance together; REST's per-molecule build
// (vk_upper_with_ri_v_sync, src/scf_io/mod.rs:2758-2834, with the J of
// vj_upper_with_rimatr_v_sync, :2490-2561) runs here for every molecule of a
// group at once.  Each phase enumerates work items over all molecules --
// (molecule, element), (molecule, aux row), (molecule, aux row, row block,
// column block), (molecule, K sub-block, split) -- and decodes the molecule
// from per-phase prefix sums in device memory.  The two tensor-core phases are
// persistent: a grid of SMs x resident CTAs walks the items.  Molecules whose
// active flag is 0 are skipped, so a captured graph serves every iteration.

__device__ __forceinline__ int group_find(const int64_t* __restrict__ pre, int count, int64_t w) {
  int lo = 0, hi = count - 1;  // largest m with pre[m] <= w
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= w)
      lo = mid;
    else
      hi = mid - 1;
  }
  return lo;
}

// Phase 1: Cw = sqrt(2) C (ldx x ocols, zero padded).
__global__ void __launch_bounds__(256) k_grp_prepare(const GroupMol* __restrict__ mols, const int64_t* __restrict__ pre,
                                                     int count, int64_t total, const double* __restrict__ C0,
                                                     int64_t c_mol, int64_t c_row, int64_t c_col,
                                                     const int* __restrict__ active) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int m = group_find(pre, count, e);
    if (!active[m]) continue;
    const GroupMol& g = mols[m];
    const double* C = C0 + m * c_mol;
    const int64_t t = e - pre[m];
    const int64_t row = t % g.ldx, col = t / g.ldx;
    g.Cw[t] = (row < g.n && col < g.nocc) ? 1.4142135623730951 * C[row * c_row + col * c_col] : 0.0;
  }
}

// Phase 3 (persistent): X_P = B_P Cw for every (molecule, aux row, row block, column block).
// XF > 0: a molecule with g.xcol0 > 0 launches only its full column blocks, and
// the CTAs of the last one also compute the XF * 8 remainder columns from xcol0
// on (ExtraCols), as the single-molecule half-transform does.
template <class Cfg, int XF = 0>
__global__ void __launch_bounds__(Cfg::THREADS, min_ctas<Cfg>()) k_grp_half(const GroupMol* __restrict__ mols,
                                                                            const int64_t* __restrict__ pre, int count,
                                                                            int64_t total, const int* __restrict__ active,
                                                                            int* err) {
  extern __shared__ __align__(128) double smem[];
  for (int64_t it = blockIdx.x; it < total; it += gridDim.x) {
    const int m = group_find(pre, count, it);
    if (!active[m]) continue;  // uniform over the CTA
    const GroupMol& g = mols[m];
    const int nrb = (int)(g.ldx / Cfg::BM), ncb = g.ncb;
    const int64_t bid = it - pre[m];
    const int cb = (int)(bid % ncb);
    const int64_t rest = bid / ncb;
    const int64_t pl = rest / nrb;
    const int I0 = (int)(rest % nrb) * Cfg::MT;
    const int col0 = cb * Cfg::BN;
    HalfTransformSched sc{g.B + pl * g.ldB, g.Cw, g.ldx, g.nt, I0, col0, g.xcol0};
    double acc[Cfg::FM][Cfg::FN][2];
    ExtraCols<XF> xc;
    xc.on = XF > 0 && g.xcol0 > 0 && cb == ncb - 1;
    const int ktiles = I0 < g.nt ? g.nt : 0;
    const LastTileK kv{g.nt - 1, g.n - (g.nt - 1) * TS};
    __syncthreads();  // the previous item's warps are done with the stages
    if (dmma_mainloop<Cfg, HalfTransformSched, LastTileK, XF>(sc, ktiles, smem, acc, err, g.n - I0 * TS,
                                                               g.nocc - col0, kv, &xc)) {
      double* Xr = g.X + (int64_t)I0 * TS;
      const double* Wr = g.Cw + (int64_t)I0 * TS;
      const int64_t nw = g.nocc;
      double s = 0.0;  // this warp's share of w_P = <Cw, X_P> = B_P : 2 C C^T
      dmma_for_each<Cfg>(acc, [&](int mm, int c, double v0, double v1) {
        const int64_t c0 = col0 + c;
        if (c0 < nw) Xr[mm + (pl * nw + c0) * g.ldx] = v0;
        if (c0 + 1 < nw) Xr[mm + (pl * nw + c0 + 1) * g.ldx] = v1;
        s = fma(v0, Wr[mm + c0 * g.ldx], s);
        s = fma(v1, Wr[mm + (c0 + 1) * g.ldx], s);
      });
      if constexpr (XF > 0) {
        if (xc.on) {
          const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
          const int wm = warp / Cfg::WN, wn = warp % Cfg::WN;
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int j = 0; j < XF; ++j) {
              const int mm = wm * Cfg::WTM + (wn * 2 + e) * 8 + (lane >> 2);
              const int64_t c = g.xcol0 + 8 * j + 2 * (lane & 3);
              const double v0 = xc.acc[e][j][0], v1 = xc.acc[e][j][1];
              if (c < nw) Xr[mm + (pl * nw + c) * g.ldx] = v0;
              if (c + 1 < nw) Xr[mm + (pl * nw + c + 1) * g.ldx] = v1;
              s = fma(v0, Wr[mm + c * g.ldx], s);
              s = fma(v1, Wr[mm + (c + 1) * g.ldx], s);
            }
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if ((threadIdx.x & 31) == 0) g.wpart[bid * Cfg::CWARPS + (threadIdx.x >> 5)] = s;
    }
  }
}

// Phase 2 (after phase 3): w_P = the warp shares of aux row P summed in a fixed
// order, one warp per (molecule, aux row).
__global__ void __launch_bounds__(256) k_grp_wreduce(const GroupMol* __restrict__ mols,
                                                     const int64_t* __restrict__ pre, int count, int64_t total,
                                                     const int* __restrict__ active) {
  const int64_t it = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (it >= total) return;
  const int m = group_find(pre, count, it);
  if (!active[m]) return;
  const GroupMol& g = mols[m];
  const int64_t P = it - pre[m];
  const double* src = g.wpart + P * g.wper;
  double a = 0.0;
  for (int t = threadIdx.x & 31; t < g.wper; t += 32) a += src[t];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if ((threadIdx.x & 31) == 0) g.w[P] = a;
}

// Phase 4 (persistent): Kpart = sum_p X_p X_p^T per (molecule, upper K sub-block, split).
template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, min_ctas<Cfg>()) k_grp_rank(const GroupMol* __restrict__ mols,
                                                                            const int64_t* __restrict__ pre, int count,
                                                                            int64_t total, const int* __restrict__ active,
                                                                            int* err) {
  extern __shared__ __align__(128) double smem[];
  constexpr int subs = (KB / Cfg::BM) * (KB / Cfg::BN);
  for (int64_t it = blockIdx.x; it < total; it += gridDim.x) {
    const int m = group_find(pre, count, it);
    if (!active[m]) continue;
    const GroupMol& g = mols[m];
    const int64_t local = it - pre[m];
    const int64_t nsub = g.pairs * subs;
    const int sp = (int)(local / nsub);
    int64_t q, row0, col0, off;
    if (!sub_block<Cfg>(local % nsub, 0, g.nkb, q, row0, col0, off)) continue;
    const int64_t pa = (int64_t)g.naux * sp / g.ksplits, pb = (int64_t)g.naux * (sp + 1) / g.ksplits;
    const int64_t kcount = (pb - pa) * g.nocc;
    RankSched sc{g.X, g.ldx, pa * g.nocc, row0, col0};
    double acc[Cfg::FM][Cfg::FN][2];
    const int ktiles = (int)((kcount + TS - 1) / TS);
    const LastTileK kv{ktiles - 1, (int)(kcount - (int64_t)(ktiles - 1) * TS)};
    __syncthreads();
    if (dmma_mainloop<Cfg>(sc, ktiles, smem, acc, err, g.n - (int)row0, g.n - (int)col0, kv)) {
      double* out = g.Kpart + ((int64_t)sp * g.pairs + q) * (KB * KB) + off;
      dmma_for_each<Cfg>(acc, [&](int mm, int c, double v0, double v1) {
        out[mm + KB * c] = v0;
        out[mm + KB * (c + 1)] = v1;
      });
    }
  }
}

// Phase 5: Jpart[split] = sum_p B[p, :] w_p per (molecule, 512-pair chunk of the row, split).
__global__ void __launch_bounds__(256) k_grp_pass2(const GroupMol* __restrict__ mols, const int64_t* __restrict__ pre,
                                                   int count, const int* __restrict__ active) {
  const int m = group_find(pre, count, blockIdx.x);
  if (!active[m]) return;
  const GroupMol& g = mols[m];
  const int64_t nq = g.ldB / 2;
  const int64_t nqb = (nq + 255) / 256;
  const int64_t local = blockIdx.x - pre[m];
  const int sp = (int)(local / nqb);
  const int64_t q = (local % nqb) * 256 + threadIdx.x;
  if (q >= nq) return;
  const int64_t p0 = (int64_t)g.naux * sp / g.jsplits, p1 = (int64_t)g.naux * (sp + 1) / g.jsplits;
  const double2* b = reinterpret_cast<const double2*>(g.B) + q;
  double2 a = make_double2(0.0, 0.0);
  for (int64_t p = p0; p < p1; ++p) {
    const double2 x = ld_stream(b + p * nq);
    const double wp = __ldg(g.w + p);
    a.x = fma(x.x, wp, a.x);
    a.y = fma(x.y, wp, a.y);
  }
  reinterpret_cast<double2*>(g.Jpart + (int64_t)sp * g.ldB)[q] = a;
}

// Phase 6: out[i, j] = out[j, i] = J_ij + k_scale K_ij (splits summed in order).
__global__ void __launch_bounds__(256) k_grp_finalize(const GroupMol* __restrict__ mols, const int64_t* __restrict__ pre,
                                                      int count, int64_t total, double* __restrict__ out0,
                                                      int64_t out_mol, int64_t ldo, double k_scale,
                                                      const int* __restrict__ active) {
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int m = group_find(pre, count, e);
    if (!active[m]) continue;
    const GroupMol& g = mols[m];
    const int64_t t = e - pre[m];
    const int64_t j = tri_root(t), i = t - j * (j + 1) / 2;
    const int64_t k = tile_pair_index(i / TS, j / TS) * TILE_ELEMS + (i % TS) + TS * (j % TS);
    double vj = 0.0;
    for (int sp = 0; sp < g.jsplits; ++sp) vj += g.Jpart[(int64_t)sp * g.ldB + k];
    const int64_t Ib = i / KB, Jb = j / KB;
    const int64_t q = Jb * (Jb + 1) / 2 + Ib;
    const int64_t off = (i % KB) + (int64_t)KB * (j % KB);
    double vk = 0.0;
    for (int sp = 0; sp < g.ksplits; ++sp) vk += g.Kpart[((int64_t)sp * g.pairs + q) * (KB * KB) + off];
    const double v = vj + k_scale * vk;
    double* o = out0 + m * out_mol;
    o[i * ldo + j] = v;
    o[j * ldo + i] = v;
  }
}

int group_ctas_per_sm(int cfg) { return cfg == 1 ? 3 : 2; }

template <class Cfg, int XF = 0>
static void grp_half_cfg(const GroupMol* mols, const int64_t* pre, int count, int64_t total, const int* active,
                         int* err, int sms, cudaStream_t st) {
  cudaFuncSetAttribute(k_grp_half<Cfg, XF>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM_BYTES);
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>(total, (int64_t)sms * min_ctas<Cfg>()));
  count_launch();
  k_grp_half<Cfg, XF><<<(unsigned)grid, Cfg::THREADS, Cfg::SMEM_BYTES, st>>>(mols, pre, count, total, active, err);
}

template <class Cfg>
static void grp_rank_cfg(const GroupMol* mols, const int64_t* pre, int count, int64_t total, const int* active,
                         int* err, int sms, cudaStream_t st) {
  cudaFuncSetAttribute(k_grp_rank<Cfg>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM_BYTES);
  const int64_t grid = std::max<int64_t>(1, std::min<int64_t>(total, (int64_t)sms * min_ctas<Cfg>()));
  count_launch();
  k_grp_rank<Cfg><<<(unsigned)grid, Cfg::THREADS, Cfg::SMEM_BYTES, st>>>(mols, pre, count, total, active, err);
}

int group_cta_rows(int cfg) { return cfg == 4 ? 128 : 64; }
int group_cta_cols(int cfg) { return 64; }
int group_rank_subs(int cfg) { return cfg == 4 ? 2 : 4; }
int group_cta_warps(int cfg) { return cfg == 4 ? HtCfg4::CWARPS : cfg == 0 ? HtCfg0::CWARPS : HtCfg1::CWARPS; }
int group_remainder_cols(int cfg) { return cfg == 1 ? 16 : 0; }

void launch_group_front(const GroupPlan& gp, const double* C0, int64_t c_mol, int64_t c_row, int64_t c_col,
                        const int* active, int* err, int sms, cudaStream_t st) {
  const int n = gp.count;
  {
    const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(gp.total[0], 256), 148 * 16));
    count_launch();
    k_grp_prepare<<<blocks, 256, 0, st>>>(gp.mols, gp.pre[0], n, gp.total[0], C0, c_mol, c_row, c_col, active);
  }
  if (gp.total[2] == 0) return;
  switch (gp.ht_cfg) {
    case 0: grp_half_cfg<HtCfg0>(gp.mols, gp.pre[2], n, gp.total[2], active, err, sms, st); break;
    case 4: grp_half_cfg<HtCfg4>(gp.mols, gp.pre[2], n, gp.total[2], active, err, sms, st); break;
    default:
      if (gp.remainder)
        grp_half_cfg<HtCfg1, 2>(gp.mols, gp.pre[2], n, gp.total[2], active, err, sms, st);
      else
        grp_half_cfg<HtCfg1>(gp.mols, gp.pre[2], n, gp.total[2], active, err, sms, st);
      break;
  }
}

void launch_group_back(const GroupPlan& gp, double k_scale, double* out0, int64_t out_mol, int64_t ldo,
                       const int* active, int* err, int sms, cudaStream_t st) {
  const int n = gp.count;
  if (gp.total[2] > 0) {
    count_launch();
    k_grp_wreduce<<<(unsigned)cdiv(gp.total[1], 8), 256, 0, st>>>(gp.mols, gp.pre[1], n, gp.total[1], active);
    switch (gp.rk_cfg) {
      case 0: grp_rank_cfg<RkCfg0>(gp.mols, gp.pre[3], n, gp.total[3], active, err, sms, st); break;
      case 4: grp_rank_cfg<RkCfg4>(gp.mols, gp.pre[3], n, gp.total[3], active, err, sms, st); break;
      default: grp_rank_cfg<RkCfg1>(gp.mols, gp.pre[3], n, gp.total[3], active, err, sms, st); break;
    }
  }
  count_launch();
  k_grp_pass2<<<(unsigned)gp.total[4], 256, 0, st>>>(gp.mols, gp.pre[4], n, active);
  {
    const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(gp.total[5], 256), 148 * 16));
    count_launch();
    k_grp_finalize<<<blocks, 256, 0, st>>>(gp.mols, gp.pre[5], n, gp.total[5], out0, out_mol, ldo, k_scale, active);
  }
}

}  // namespace rijk

#include <atomic>
namespace rijk {
static std::atomic<int64_t> g_launches{0};
void count_launch(int64_t k) { g_launches.fetch_add(k, std::memory_order_relaxed); }
int64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }
}  // namespace rijk

// ============================================================================
// ri3mo (ao2mo_rayon, src/scf_io/mod.rs:3270-3307)
// ============================================================================
namespace rijk {

// out (ldo x ncp, zero padded) = C[:, c0 : c0 + nc]  (C column-major, ld = ldc_in)
__global__ void __launch_bounds__(256) k_gather_cols(const double* __restrict__ C, int64_t n, int64_t ldc_in,
                                                     int64_t c0, int64_t nc, int64_t ldo, int64_t ncp,
                                                     double* __restrict__ out) {
  const int64_t total = ldo * ncp;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = e % ldo, c = e / ldo;
    out[e] = (r < n && c < nc) ? C[r + ldc_in * (c0 + c)] : 0.0;
  }
}

void launch_gather_cols(const double* C, int64_t n, int64_t ldc_in, int64_t c0, int64_t nc, int64_t ldo, int64_t ncp,
                        double* out, cudaStream_t st) {
  const int64_t total = ldo * ncp;
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(total, 256), 148 * 16));
  count_launch();
  k_gather_cols<<<blocks, 256, 0, st>>>(C, n, ldc_in, c0, nc, ldo, ncp, out);
}

// ri3mo[p + naux (a + nrow i)] = Y[p][a + ldy i] for the P chunk [p0, p0 + np)
__global__ void __launch_bounds__(256) k_ri3mo_permute(const double* __restrict__ Y, int64_t ldy, int64_t sy,
                                                       int64_t np, int64_t nrow, int64_t ncol,
                                                       double* __restrict__ out) {
  // out is the chunk buffer [np][nrow * ncol] with p fastest: out[p + np (a + nrow i)]
  const int64_t total = np * nrow * ncol;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = e % np, ai = e / np;
    const int64_t a = ai % nrow, i = ai / nrow;
    out[e] = Y[p * sy + a + ldy * i];
  }
}

void launch_ri3mo_permute(const double* Y, int64_t ldy, int64_t sy, int64_t np, int64_t nrow, int64_t ncol,
                          double* out, cudaStream_t st) {
  const int64_t total = np * nrow * ncol;
  const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(cdiv(total, 256), 148 * 32));
  count_launch();
  k_ri3mo_permute<<<blocks, 256, 0, st>>>(Y, ldy, sy, np, nrow, ncol, out);
}

}  // namespace rijk
