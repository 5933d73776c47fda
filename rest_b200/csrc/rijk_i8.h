// Host-side launchers of the FP64 contractions that run on the INT8 tensor
// cores (rijk_i8.cu), internal to librest_b200.so.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace rijk {

constexpr int I8_DIGITS = 7;  // base-256 digits of an operand
// A level sums at most seven digit products of 2^14 per element of the contracted index:
// this many stay below 2^31 (the half-transform contracts over the basis functions).
constexpr int64_t I8_MAX_N = 16384;

// `active` of the launches below: null, or a device flag; where it is 0 the kernel
// does nothing (a group's converged molecules in a captured graph).  Groups take the
// in-tile half-transform only, and only that form of launch_i8_half looks at it.

// Digits of a column-major FP64 matrix X (ldx rows, ldx a multiple of 128, k
// columns): for every group of 16 columns, digit and row the 16 digits of that
// row, zero beyond column k.
inline int64_t i8_groups(int64_t k) { return (k + 15) / 16; }
inline int64_t i8_digit_bytes(int64_t ldx, int64_t k) { return i8_groups(k) * I8_DIGITS * ldx * 16; }
// maxhi[row] = the high word of the largest |X[row, :]|
void launch_i8_slice(const double* X, int64_t ldx, int64_t k, const int* maxhi, int8_t* digits, cudaStream_t st,
                     const int* active = nullptr);

// Splits of the k range the update takes (scratch: splits x pairs x 128 x 128 doubles).
int i8_rank_splits(int64_t n, int64_t k, int full);
// Kpart[split][q] (128 x 128 blocks q over block pairs, as launch_k_rank_update
// writes them) = the split's share of X Y^T for the digit matrices X and Y (ldx
// rows, k columns each; xmax and ymax their rows' maxima, as maxhi above).  full = 0: the
// blocks' upper triangle only.  False when the operands' tensor maps could not be encoded:
// nothing is launched then.
bool launch_i8_rank(int64_t n, int64_t ldx, int64_t k, const int8_t* xdig, const int* xmax, const int8_t* ydig,
                    const int* ymax, int splits, int full, double* Kpart, int* err, cudaStream_t st,
                    const int* active = nullptr);

// --- half-transform X_P = B_P C on the INT8 tensor cores -----------------------
// Columns are padded per spin to groups of 16 (spin 1 after spin 0).
struct I8Cols {
  int64_t nw[2] = {0, 0};  // orbitals per spin
  int g[2] = {0, 0};       // their 16-column groups
  int cols() const { return 16 * (g[0] + g[1]); }
};
I8Cols i8_cols(const int64_t* nw, int spin);
// column blocks (of at most 64 columns) a row block's orbitals take
int i8_blocks(const I8Cols& c);
// bmax[P ldx + row] = the high word of the largest |B_P[row, :]| (rows below ldx)
void launch_i8_tensor_max(const double* B, int64_t ldB, int64_t nt, int64_t naux, int64_t ldx, int* bmax,
                          cudaStream_t st);
// Orbitals scaled by sqrt(occupation) (occ null: as they are): Cw (ldx x cols,
// zero padded), their digits (i8_col_bytes) and each column's result factor; columns
// from `valid` of a spin on are zero.
int64_t i8_col_bytes(const I8Cols& c, int64_t nt);
void launch_i8_cols(const I8Cols& c, const double* eigv, int64_t n, int64_t nt, int64_t ldx, int64_t ld_eigv,
                    int64_t stride_eigv, const double* occ, int64_t stride_occ, double* Cw, int8_t* digits,
                    double* factor, int* err, cudaStream_t st, int valid = 1 << 30);
// Whether a row block's digits are made where they are used: the half-transform
// then reads I8Chunk::B and needs no digits, and I8Next has to be empty.
bool i8_in_tile(const I8Cols& c);
// The half-transform of one chunk of aux rows from its tensor digits, and the
// tensor digits of the next chunk (either may be empty: np = 0).
struct I8Chunk {
  int64_t np = 0;
  const double* B = nullptr;       // tile-packed rows, stride ldB
  const int8_t* digits = nullptr;  // i8_row_bytes per aux row
  const int* bmax = nullptr;       // at the chunk's first aux row, as its digits and the following
  double* X[2] = {nullptr, nullptr};  // per spin: X_p's nw columns (ldx rows) back to back
  double* wpart = nullptr;            // shares of J's scalars (np x i8_wpart_rows x 2 doubles), or null
};
struct I8Next {
  int64_t np = 0;
  const double* B = nullptr;
  const int* bmax = nullptr;
  bool shared_max = false;  // bmax holds one row of maxima for all of the chunk's aux rows
  int8_t* digits = nullptr;
};
void launch_i8_max_rows(const int* bmax, int64_t ldx, int64_t np, int* cmax, cudaStream_t st);
int64_t i8_row_bytes(int64_t nt, int64_t ldx);
int64_t i8_chunk_rows(const I8Cols& c, int64_t nt, int64_t ldx, int64_t naux, int64_t bytes);
// xmax[spin ldx + row] takes the high word of the largest |X[row, :]| (the caller clears it).
// False as launch_i8_rank's.
bool launch_i8_half(const I8Cols& c, int64_t n, int64_t nt, int64_t ldx, int64_t ldB, const I8Chunk& cur,
                    const I8Next& next, const double* Cw, const int8_t* digits, const double* factor, int* xmax, int* err,
                    cudaStream_t st, const int* active = nullptr);
// per-warp shares of J's scalars per aux row, for launch_j_wreduce
int64_t i8_wpart_rows(const I8Cols& c, int64_t ldx);
// w[s][p0 + p] = the sum, in a fixed order, of aux row p's per_row pairs of shares
void launch_j_wreduce(const double* wpart, int64_t np, int per_row, int nspin, int64_t naux, int64_t p0, double* w,
                      cudaStream_t st);
}  // namespace rijk
