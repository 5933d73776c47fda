// Kernels of the learned initial guess: a per-atom-pair MLP with BF16 weights
// and activations and FP32 accumulation, trained and evaluated on the device.
// REST has no learned guess; its own guesses (src/initial_guess) stay the
// fallback of the driver that uses this network.
//
//   linear forward   Z = X W^T + b, Y = act(Z)      (X: m x k, W: n x k, row-major)
//   linear backward  dZ = dY * act'(Z), db = sum_m dZ (FP32), dW = dZ^T X, dX = dZ W (dZ as BF16)
//   masked MSE       loss += sum mask (Y - T)^2 / count, dY = 2 mask (Y - T) / count
//   Adam             FP32 master weights, BF16 copies written back
//
// The GEMMs run on the tensor cores: BF16 operands staged in shared memory,
// mma.sync m16n8k16 with FP32 accumulation, 64 x 64 CTA tiles of four warps
// (32 x 32 each), k-step 32; operands contiguous in either index (X W^T, dZ^T X, dZ W).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/rest_b200.h"
#include "rijk_internal.h"

namespace {

constexpr int NT = 256;                 // threads of the elementwise kernels
constexpr int TM = 64, TN = 64, TK = 32;  // GEMM CTA tile and k-step
constexpr int GT = 128;                 // GEMM threads: 4 warps of 32 x 32
constexpr int SK = TK + 8;              // smem row of an l-contiguous tile (BF16): 80 bytes, conflict-free fragment loads

__device__ __forceinline__ uint16_t to_bf(float v) { return __bfloat16_as_ushort(__float2bfloat16_rn(v)); }

__device__ __forceinline__ float act_f(int act, float z) { return act == 1 ? z / (1.0f + expf(-z)) : z; }
__device__ __forceinline__ float act_d(int act, float z) {
  if (act != 1) return 1.0f;
  const float s = 1.0f / (1.0f + expf(-z));
  return s + z * s * (1.0f - s);
}

// D(16x8) += A(16x16, row) B(16x8, col), BF16 in, FP32 accumulate.
__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// One operand of the GEMM: 64 rows (of A, or columns of B) by TK of the inner
// index, X(row, l) at p[row * sr + l * sl] where one of the strides is 1.  Its tile
// lies in shared memory with the contiguous index along the rows (l: rows of SK;
// row: rows of SR), filled from registers that a step ahead were loaded in runs of
// VEC elements: 8 or 4 where the other stride and the address allow 16- or 8-byte
// loads, else 1.
constexpr int SR = TM + 8;  // smem row of a row-contiguous tile: conflict-free transposing loads

struct Operand {
  const uint16_t* p;
  int64_t stride;  // of the index that is not contiguous
  int64_t rows;    // limit of the row index
  bool by_l;       // l is the contiguous index
  int vec;
};

// This thread's 16 elements of the tile at (row0, l0): 16 / VEC runs of VEC along the contiguous index.
template <int VEC>
__device__ __forceinline__ void load_tile(const Operand& o, int64_t row0, int64_t l0, int64_t l_end,
                                          uint32_t (&v)[8]) {
  constexpr int RUNS = 16 / VEC;
#pragma unroll
  for (int u = 0; u < RUNS; ++u) {
    const int e = (threadIdx.x + GT * u) * VEC;
    const int inner = o.by_l ? TK : TM;
    const int c = e % inner, other = e / inner;
    const int64_t row = row0 + (o.by_l ? other : c), l = l0 + (o.by_l ? c : other);
    const uint16_t* src = o.p + (o.by_l ? row * o.stride + l : l * o.stride + row);
    if constexpr (VEC == 1) {
      uint32_t x = (row < o.rows && l < l_end) ? (uint32_t)__ldg(src) : 0u;
      if (u & 1)
        v[u >> 1] |= x << 16;
      else
        v[u >> 1] = x;
    } else {
      // runs start at multiples of VEC of a stride and limits that are multiples of VEC
      const bool in = row < o.rows && l < l_end;
      if constexpr (VEC == 8) {
        const uint4 x = in ? __ldg(reinterpret_cast<const uint4*>(src)) : make_uint4(0, 0, 0, 0);
        v[4 * u] = x.x, v[4 * u + 1] = x.y, v[4 * u + 2] = x.z, v[4 * u + 3] = x.w;
      } else {
        const uint2 x = in ? __ldg(reinterpret_cast<const uint2*>(src)) : make_uint2(0, 0);
        v[2 * u] = x.x, v[2 * u + 1] = x.y;
      }
    }
  }
}

template <int VEC>
__device__ __forceinline__ void store_tile(const Operand& o, const uint32_t (&v)[8], uint16_t* sm) {
  constexpr int RUNS = 16 / VEC;
#pragma unroll
  for (int u = 0; u < RUNS; ++u) {
    const int e = (threadIdx.x + GT * u) * VEC;
    const int inner = o.by_l ? TK : TM;
    uint16_t* d = sm + (e / inner) * (o.by_l ? SK : SR) + e % inner;
    if constexpr (VEC == 8)
      *reinterpret_cast<uint4*>(d) = make_uint4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
    else if constexpr (VEC == 4)
      *reinterpret_cast<uint2*>(d) = make_uint2(v[2 * u], v[2 * u + 1]);
    else
      *d = (uint16_t)(v[u >> 1] >> (16 * (u & 1)));
  }
}

__device__ __forceinline__ void load_tile(const Operand& o, int64_t row0, int64_t l0, int64_t l_end,
                                          uint32_t (&v)[8]) {
  if (o.vec == 8)
    load_tile<8>(o, row0, l0, l_end, v);
  else if (o.vec == 4)
    load_tile<4>(o, row0, l0, l_end, v);
  else
    load_tile<1>(o, row0, l0, l_end, v);
}
__device__ __forceinline__ void store_tile(const Operand& o, const uint32_t (&v)[8], uint16_t* sm) {
  if (o.vec == 8)
    store_tile<8>(o, v, sm);
  else if (o.vec == 4)
    store_tile<4>(o, v, sm);
  else
    store_tile<1>(o, v, sm);
}

// Four 8 x 8 fragments, each from the 16-byte rows that 8 lanes address.
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const uint16_t* p, bool trans) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  if (trans)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}
// Rows row .. row + 15, l .. l + 15 of a tile as {rows 0-7 l 0-7, rows 8-15 l 0-7, rows 0-7 l 8-15, rows 8-15 l 8-15}.
__device__ __forceinline__ void frag16(uint32_t (&r)[4], const Operand& o, const uint16_t* sm, int row, int l, int lane) {
  if (o.by_l)
    ldsm4(r, sm + (row + (lane & 15)) * SK + l + 8 * (lane >> 4), false);
  else
    ldsm4(r, sm + (l + (lane & 7) + 8 * (lane >> 4)) * SR + row + 8 * ((lane >> 3) & 1), true);
}

// C[i, j] = sum_l A(i, l) B(j, l) over l in this CTA's k-chunk; tiles two deep in
// shared memory, the next one's loads in flight behind the MMAs.  Loaded two bytes at
// a time and waited for at each step, the same tiles took 449 of 659 us of kernel time
// of a training step on 4096 rows (one kernel after another under the profiler); the
// step itself went from 560 to 321 us with this form and the activation kernel below.
// EPI 0: forward epilogue (bias, activation, Z / Ybf / Yf outputs, no split-k);
// EPI 1: plain FP32 output, atomically added (split-k over blockIdx.z); EPI 2: stored.
template <int EPI>
__global__ void __launch_bounds__(GT) k_gemm(int64_t M, int64_t N, int64_t K, int64_t kchunk, Operand A, Operand B,
                                             const float* __restrict__ bias, int act, float* __restrict__ Z,
                                             uint16_t* __restrict__ Ybf, float* __restrict__ Yf,
                                             float* __restrict__ C) {
  constexpr int TILE = TM * SK > TK * SR ? TM * SK : TK * SR;
  __shared__ __align__(16) uint16_t As[2][TILE];
  __shared__ __align__(16) uint16_t Bs[2][TILE];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp >> 1, wn = warp & 1;  // warp tile rows wm*32, cols wn*32
  const int64_t i0 = (int64_t)blockIdx.y * TM, j0 = (int64_t)blockIdx.x * TN;
  const int64_t l_begin = (int64_t)blockIdx.z * kchunk;
  const int64_t l_end = l_begin + kchunk < K ? l_begin + kchunk : K;
  float acc[2][4][4] = {};
  const int q = lane >> 2, r = lane & 3;
  uint32_t va[8], vb[8];
  load_tile(A, i0, l_begin, l_end, va);
  load_tile(B, j0, l_begin, l_end, vb);
  int st = 0;
  for (int64_t l0 = l_begin; l0 < l_end; l0 += TK, st ^= 1) {
    store_tile(A, va, As[st]);
    store_tile(B, vb, Bs[st]);
    __syncthreads();  // the tile is there; the other one's readers are two steps behind
    if (l0 + TK < l_end) {
      load_tile(A, i0, l0 + TK, l_end, va);
      load_tile(B, j0, l0 + TK, l_end, vb);
    }
#pragma unroll
    for (int k0 = 0; k0 < TK; k0 += 16) {
      uint32_t af[2][4], bq[2][4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) frag16(af[mt], A, As[st], wm * 32 + mt * 16, k0, lane);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) frag16(bq[nt], B, Bs[st], wn * 32 + nt * 16, k0, lane);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const uint32_t bf[2] = {bq[nt >> 1][nt & 1], bq[nt >> 1][2 + (nt & 1)]};
          mma_bf16_16816(acc[mt][nt], af[mt], bf);
        }
    }
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t i = i0 + wm * 32 + mt * 16 + q + 8 * h;
      if (i >= M) continue;
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int64_t j = j0 + wn * 32 + nt * 8 + 2 * r + e;
          if (j >= N) continue;
          const float v = acc[mt][nt][2 * h + e];
          if (EPI == 0) {
            const float z = v + (bias ? bias[j] : 0.0f);
            if (Z) Z[i * N + j] = z;
            const float y = act_f(act, z);
            if (Ybf) Ybf[i * N + j] = to_bf(y);
            if (Yf) Yf[i * N + j] = y;
          } else if (EPI == 1) {
            atomicAdd(&C[i * N + j], v);
          } else {
            C[i * N + j] = v;
          }
        }
    }
}

// The widest load an operand allows: its stride, its limits and (with the chunks'
// starts) its address have to be multiples of it.
Operand operand(const uint16_t* p, int64_t rows, int64_t inner, int64_t stride, bool by_l) {
  Operand o{p, stride, rows, by_l, 1};
  const int64_t all = stride | (by_l ? inner : rows) | (int64_t)(reinterpret_cast<uintptr_t>(p) / 2);
  if ((reinterpret_cast<uintptr_t>(p) & 1) == 0) o.vec = all % 8 == 0 ? 8 : all % 4 == 0 ? 4 : 1;
  return o;
}

// dZ = dY * act'(Z) as BF16, and db += column sums.  A CTA takes 64 rows of 64
// columns, four groups of threads 16 rows each (one thread per column of the 64 rows
// left half of the GPU idle: 33 us at 4096 x 256).
constexpr int AR = 64, AC = 64;
__global__ void __launch_bounds__(NT) k_act_bwd(int64_t M, int64_t N, const float* __restrict__ dY,
                                                const float* __restrict__ Z, int act, uint16_t* __restrict__ dZ,
                                                float* __restrict__ db) {
  __shared__ float part[NT];
  const int64_t j = (int64_t)blockIdx.y * AC + threadIdx.x % AC;
  constexpr int ROWS = AR / (NT / AC);
  const int64_t r0 = (int64_t)blockIdx.x * AR + threadIdx.x / AC * ROWS;
  float s = 0.0f;
  if (j < N) {
#pragma unroll 4
    for (int64_t i = r0; i < (r0 + ROWS < M ? r0 + ROWS : M); ++i) {
      const float g = dY[i * N + j] * act_d(act, Z[i * N + j]);
      dZ[i * N + j] = to_bf(g);
      s += g;
    }
  }
  if (!db) return;
  part[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x < AC && j < N) {
    for (int q = AC; q < NT; q += AC) s += part[threadIdx.x + q];
    atomicAdd(&db[j], s);
  }
}

__global__ void __launch_bounds__(NT) k_masked_mse(int64_t count, const float* __restrict__ Y,
                                                   const float* __restrict__ T, const float* __restrict__ mask,
                                                   float inv_n, float* __restrict__ dY, float* __restrict__ loss) {
  __shared__ float red[NT];
  float s = 0.0f;
  for (int64_t e = (int64_t)blockIdx.x * NT + threadIdx.x; e < count; e += (int64_t)gridDim.x * NT) {
    const float mk = mask ? mask[e] : 1.0f;
    const float d = (Y[e] - T[e]) * mk;
    dY[e] = 2.0f * d * inv_n;
    s += d * d;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = NT / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0 && loss) atomicAdd(loss, red[0] * inv_n);
}

__global__ void __launch_bounds__(NT) k_adam(int64_t count, float* __restrict__ w, uint16_t* __restrict__ wbf,
                                             const float* __restrict__ g, float* __restrict__ m,
                                             float* __restrict__ v, float lr, float b1, float b2, float eps,
                                             float bc1, float bc2) {
  for (int64_t e = (int64_t)blockIdx.x * NT + threadIdx.x; e < count; e += (int64_t)gridDim.x * NT) {
    const float ge = g[e];
    const float me = b1 * m[e] + (1.0f - b1) * ge;
    const float ve = b2 * v[e] + (1.0f - b2) * ge * ge;
    m[e] = me;
    v[e] = ve;
    const float we = w[e] - lr * (me / bc1) / (sqrtf(ve / bc2) + eps);
    w[e] = we;
    if (wbf) wbf[e] = to_bf(we);
  }
}

__global__ void __launch_bounds__(NT) k_to_bf16(int64_t count, const float* __restrict__ s, uint16_t* __restrict__ d) {
  for (int64_t e = (int64_t)blockIdx.x * NT + threadIdx.x; e < count; e += (int64_t)gridDim.x * NT)
    d[e] = to_bf(s[e]);
}

// Learned-guess density assembly (the inverse of the training targets' frame
// rotation).  Unordered atom pair u (A <= B, within the cutoff) is
// up[4u .. 4u+3] = (A, B, ordered pair index of (A, B), of (B, A)) into the
// network output y (standardised, 196 per pair: the 14 x 14 block, row-major).
// With P = y t_std[kind] + t_mean[kind] (kind = 2 type(A) + type(B)) and G_t(w)
// the rotation of element t's AO block into water w's frame (rot, 14 x 14 per
// water and element, row-major):
//   D_AB = 1/2 (G_tA(wA) P_AB G_tB(wA)^T + G_tA(wB) P_BA^T G_tB(wB)^T),
// the average of the (A, B) prediction and the transposed (B, A) one, each
// rotated back from its own water's frame.  D_AB and D_BA = D_AB^T are written
// once each (no atomics); one warp per pair.
constexpr int GB = 14, GB2 = GB * GB;

__global__ void __launch_bounds__(128) k_guess_assemble(const float* __restrict__ y, const float* __restrict__ t_mean,
                                                        const float* __restrict__ t_std, const int32_t* __restrict__ up,
                                                        int64_t nu, const int32_t* __restrict__ first,
                                                        const int32_t* __restrict__ type,
                                                        const int32_t* __restrict__ nfun,
                                                        const int32_t* __restrict__ water,
                                                        const double* __restrict__ rot, int64_t n,
                                                        double* __restrict__ D) {
  __shared__ double sm[4][4][GB2];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  double* P1 = sm[wl][0];   // P_AB            (na x nb)
  double* P2 = sm[wl][1];   // P_BA^T          (na x nb)
  double* T1 = sm[wl][2];   // P_AB G_tB(wA)^T (na x nb)
  double* T2 = sm[wl][3];   // P_BA^T G_tB(wB)^T
  for (int64_t u = (int64_t)blockIdx.x * 4 + wl; u < nu; u += (int64_t)gridDim.x * 4) {
    const int a = up[4 * u], b = up[4 * u + 1];
    const int64_t iab = up[4 * u + 2], iba = up[4 * u + 3];
    const int ta = type[a], tb = type[b], na = nfun[a], nb = nfun[b];
    if (na > GB || nb > GB || na < 0 || nb < 0 || (ta | tb) & ~1) continue;  // outside the 14 x 14 blocks: skipped
    const int kab = 2 * ta + tb, kba = 2 * tb + ta;
    const double* GAa = rot + ((int64_t)water[a] * 2 + ta) * GB2;
    const double* GBa = rot + ((int64_t)water[a] * 2 + tb) * GB2;
    const double* GAb = rot + ((int64_t)water[b] * 2 + ta) * GB2;
    const double* GBb = rot + ((int64_t)water[b] * 2 + tb) * GB2;
    for (int e = lane; e < GB2; e += 32) {
      const int r = e / GB, c = e % GB;
      double p1 = 0.0, p2 = 0.0;
      if (r < na && c < nb) {
        p1 = (double)(y[iab * GB2 + e] * t_std[kab * GB2 + e] + t_mean[kab * GB2 + e]);
        const int et = c * GB + r;  // (c, r) of the (B, A) block
        p2 = (double)(y[iba * GB2 + et] * t_std[kba * GB2 + et] + t_mean[kba * GB2 + et]);
      }
      P1[e] = p1;
      P2[e] = p2;
    }
    __syncwarp();
    for (int e = lane; e < GB2; e += 32) {
      const int r = e / GB, c = e % GB;
      double s1 = 0.0, s2 = 0.0;
      if (r < na && c < nb)
        for (int k = 0; k < nb; ++k) {
          s1 += P1[r * GB + k] * GBa[c * GB + k];
          s2 += P2[r * GB + k] * GBb[c * GB + k];
        }
      T1[e] = s1;
      T2[e] = s2;
    }
    __syncwarp();
    const int64_t fa = first[a], fb = first[b];
    for (int e = lane; e < GB2; e += 32) {
      const int r = e / GB, c = e % GB;
      // a diagonal block (A = B) is written from its upper triangle only, both
      // positions with one value, so the density is exactly symmetric
      if (r < na && c < nb && (a != b || r <= c)) {
        double s = 0.0;
        for (int k = 0; k < na; ++k) s += GAa[r * GB + k] * T1[k * GB + c] + GAb[r * GB + k] * T2[k * GB + c];
        if (a == b)  // average the two rounding-level different halves
          for (int k = 0; k < na; ++k) s += GAa[c * GB + k] * T1[k * GB + r] + GAb[c * GB + k] * T2[k * GB + r];
        s *= a == b ? 0.25 : 0.5;
        D[(fa + r) * n + fb + c] = s;
        D[(fb + c) * n + fa + r] = s;
      }
    }
    __syncwarp();
  }
}

unsigned grid_for(int64_t count) {
  const int64_t b = (count + NT - 1) / NT;
  return (unsigned)(b < 148 * 16 ? (b > 0 ? b : 1) : 148 * 16);
}

int launch_status() { return cudaGetLastError() == cudaSuccess ? RIJK_OK : RIJK_ERR_CUDA; }

}  // namespace

extern "C" {

int rijk_mlp_linear_fwd(const uint16_t* x, const uint16_t* w, const float* bias, int64_t m, int64_t k, int64_t n,
                        int act, float* z, uint16_t* y_bf16, float* y_f32, void* stream) {
  if (!x || !w || m <= 0 || k <= 0 || n <= 0 || (act != 0 && act != 1) || (!z && !y_bf16 && !y_f32))
    return RIJK_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 grid((unsigned)((n + TN - 1) / TN), (unsigned)((m + TM - 1) / TM), 1);
  rijk::count_launch();
  k_gemm<0><<<grid, GT, 0, st>>>(m, n, k, k, operand(x, m, k, k, true), operand(w, n, k, k, true), bias, act, z,
                                 y_bf16, y_f32, nullptr);
  return launch_status();
}

int rijk_mlp_linear_bwd(const uint16_t* x, const uint16_t* w, const float* z, const float* dy, int64_t m, int64_t k,
                        int64_t n, int act, uint16_t* dz_scratch, float* dw, float* db, float* dx, void* stream) {
  if (!x || !w || !z || !dy || !dz_scratch || !dw || m <= 0 || k <= 0 || n <= 0 || (act != 0 && act != 1))
    return RIJK_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(dw, 0, (size_t)n * k * sizeof(float), st) != cudaSuccess) return RIJK_ERR_CUDA;
  if (db && cudaMemsetAsync(db, 0, (size_t)n * sizeof(float), st) != cudaSuccess) return RIJK_ERR_CUDA;
  rijk::count_launch();
  k_act_bwd<<<dim3((unsigned)((m + AR - 1) / AR), (unsigned)((n + AC - 1) / AC)), NT, 0, st>>>(m, n, dy, z, act,
                                                                                               dz_scratch, db);
  // dW[n x k] = dZ^T X: inner dimension m, split over blockIdx.z
  {
    const int64_t tiles = ((n + TM - 1) / TM) * ((k + TN - 1) / TN);
    int64_t splits = (4 * 148 + tiles - 1) / tiles;
    int64_t kchunk = (m + splits - 1) / splits;
    kchunk = (kchunk + TK - 1) / TK * TK;
    splits = (m + kchunk - 1) / kchunk;
    const dim3 grid((unsigned)((k + TN - 1) / TN), (unsigned)((n + TM - 1) / TM), (unsigned)splits);
    rijk::count_launch();
    k_gemm<1><<<grid, GT, 0, st>>>(n, k, m, kchunk, operand(dz_scratch, n, m, n, false), operand(x, k, m, k, false),
                                   nullptr, 0, nullptr, nullptr, nullptr, dw);
  }
  // dX[m x k] = dZ W: inner dimension n
  if (dx) {
    const dim3 grid((unsigned)((k + TN - 1) / TN), (unsigned)((m + TM - 1) / TM), 1);
    rijk::count_launch();
    k_gemm<2><<<grid, GT, 0, st>>>(m, k, n, n, operand(dz_scratch, m, n, n, true), operand(w, k, n, k, false), nullptr,
                                   0, nullptr, nullptr, nullptr, dx);
  }
  return launch_status();
}

int rijk_mlp_masked_mse(const float* y, const float* t, const float* mask, int64_t count, double norm, float* dy,
                        float* loss, void* stream) {
  if (!y || !t || !dy || count <= 0 || !(norm > 0.0)) return RIJK_ERR_ARG;
  rijk::count_launch();
  k_masked_mse<<<grid_for(count), NT, 0, static_cast<cudaStream_t>(stream)>>>(count, y, t, mask,
                                                                              (float)(1.0 / norm), dy, loss);
  return launch_status();
}

int rijk_mlp_adam(float* w, uint16_t* w_bf16, const float* g, float* m, float* v, int64_t count, double lr,
                  double beta1, double beta2, double eps, int64_t step, void* stream) {
  if (!w || !g || !m || !v || count <= 0 || step <= 0) return RIJK_ERR_ARG;
  const double bc1 = 1.0 - pow(beta1, (double)step), bc2 = 1.0 - pow(beta2, (double)step);
  rijk::count_launch();
  k_adam<<<grid_for(count), NT, 0, static_cast<cudaStream_t>(stream)>>>(
      count, w, w_bf16, g, m, v, (float)lr, (float)beta1, (float)beta2, (float)eps, (float)bc1, (float)bc2);
  return launch_status();
}

int rijk_guess_assemble(const float* y, const float* t_mean, const float* t_std, const int32_t* upairs,
                        int64_t npairs, const int32_t* atom_first, const int32_t* atom_type, const int32_t* atom_nfun,
                        const int32_t* atom_water, const double* rot, int64_t num_basis, double* dm, void* stream) {
  if (!y || !t_mean || !t_std || !upairs || !atom_first || !atom_type || !atom_nfun || !atom_water || !rot || !dm ||
      npairs < 0 || num_basis <= 0)
    return RIJK_ERR_ARG;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(dm, 0, (size_t)num_basis * num_basis * sizeof(double), st) != cudaSuccess) return RIJK_ERR_CUDA;
  if (npairs == 0) return RIJK_OK;
  const unsigned blocks = (unsigned)std::min<int64_t>((npairs + 3) / 4, 148 * 16);
  rijk::count_launch();
  k_guess_assemble<<<blocks, 128, 0, st>>>(y, t_mean, t_std, upairs, npairs, atom_first, atom_type, atom_nfun,
                                           atom_water, rot, num_basis, dm);
  return launch_status();
}

int rijk_mlp_to_bf16(const float* src, uint16_t* dst, int64_t count, void* stream) {
  if (!src || !dst || count <= 0) return RIJK_ERR_ARG;
  rijk::count_launch();
  k_to_bf16<<<grid_for(count), NT, 0, static_cast<cudaStream_t>(stream)>>>(count, src, dst);
  return launch_status();
}

}  // extern "C"
