// Kernel declarations of the RI-GW engine.
#pragma once
#include "common.cuh"
#include "dgemm_mn.cuh"
#include "problem.cuh"

namespace rigw {

// Generic work-list entry of the non-GEMM kernels: problem index + up to three
// kernel-specific integers.
struct WorkItem {
  int prob, a, b, c;
};

__global__ void pack_m_kernel(const ProbDev* probs, const WorkItem* items);
__global__ void init_rhs_kernel(const ProbDev* probs, const WorkItem* items);
__global__ void mnorm_kernel(const ProbDev* probs, const WorkItem* items);
constexpr int kDiagThreads = 256;  // threads of chol_diag_kernel
__global__ void chol_diag_kernel(const ProbDev* probs, const WorkItem* items, int k);
size_t chol_diag_smem_bytes();   // dynamic shared memory of chol_diag_kernel
__global__ void energy_kernel(const ProbDev* probs, const WorkItem* items);
__global__ void trace_kernel(const ProbDev* probs, const WorkItem* items);
__global__ void pad_eps_kernel(const ProbDev* probs, const WorkItem* items);
__global__ void vchiv_kernel(const ProbDev* probs, const WorkItem* items);
__global__ void sigma_kernel(const ProbDev* probs, const WorkItem* items);
__global__ void pade_qp_kernel(const ProbDev* probs, const WorkItem* items);
__global__ void energy_sum_kernel(const ProbDev* probs, int nprob);

// AO -> MO transform helpers (kernels_aomo.cu).
struct AomoUnpackItem {
  const double* eri3;     // [naux][npair] pair-packed, diagonal x0.5
  const int* index_basis; // [npair][2] 1-based
  double* bfull;          // [nbf][nbf][naux_pad]
  int naux, naux_pad, npair, nbf, p0;
};
__global__ void aomo_unpack_kernel(AomoUnpackItem it);
// out[r][p0 + P] = src[(n, m)][P]: rows r = n mc + m of naux entries from a chunk [n][mcp][pcp].
__global__ void aomo_store_kernel(const double* src, double* out, int mc, int mcp, int pcp, int cnt, long long naux);

// One 128 x 128 tile of a general tensor-core product A B^T of the AO->MO transform
// (syrk_bf16x3.cu, syrk_ozaki.cu).
struct TcItem {
  const void* tmap;     // CUtensorMap of A: rows of 128 bytes along K
  const void* tmap_b;   // of B
  double* C;
  int* err;
  int row_a, row_b;     // tensor rows of the hi planes (Ozaki: first slices)
  int lo_off, lo_off_b; // rows from a plane to the next
  int ktiles;           // k-tiles of 64 bf16 or 128 int8
  int ldc;
  const int* ea;        // Ozaki: row exponents of A and B
  const int* eb;
  int slices;
  int mrows, ncols;     // rows and columns stored
};
// Split of a general FP64 operand into K-major bf16 hi/lo for the tensor-core
// kernel: element (r, k) of batch z is src[z*zs_src + r*rs + k*ks]; dst holds
// [2][Rpad][Kpad] per batch (hi rows, then lo rows), zero padded.
struct SplitOp {
  const double* src;
  long long rs, ks, zs_src;
  int R, K, Rpad, Kpad, nz;
  void* dst;
  long long zs_dst;   // elements between batches of dst
};
void launch_split_kmajor(const SplitOp& op, cudaStream_t s);
// Ozaki slicing of a general FP64 operand: element (r, k) of batch z is
// src[z*zs_src + r*rs + k*ks]; row r is scaled by 2^-e_r (e_r the exponent of
// max_k |x_rk|, to exps[z*Rpad + r]) and cut into `slices` int8 base-128 digits,
// stored K-contiguous as [nz][slices][Rpad][Kpad] (Kpad a multiple of 128, zero
// padded).  rmax is [nz][Rpad] scratch.
struct SliceOp {
  const double* src;
  long long rs, ks, zs_src;
  int R, K, Rpad, Kpad, nz, slices;
  void* dst;
  unsigned long long* rmax;
  int* exps;
};
void launch_slice_kmajor(const SliceOp& op, cudaStream_t s);
void launch_syrk_bf16x3(const TcItem* items, int n, cudaStream_t s);
void launch_syrk_ozaki(const TcItem* items, int n, cudaStream_t s);
cudaError_t prepare_ozaki_kernels();
cudaError_t prepare_tc_kernels();

// FP64 chi0 with TMA-staged operands (syrk_f64_tma.cu): one 64 x 128 upper tile
// of eps(iw) = 1 + sum_t M[t][i] D_w(t) M[t][j] per CTA, frequency = blockIdx.y.
struct F64SyrkItem {
  const void* tmap_m;   // CUtensorMap of mp [nia_pad][npad] (16 x 16 boxes, 128-byte swizzle)
  const void* tmap_d;   // CUtensorMap of dscale [nomega][nia_pad] (16 x 1 boxes)
  double* C;            // &eps[0][ti][tj]
  int* err;
  const int* only_if;   // run only when set (negative factors, which the digits do not take); nullptr: always
  int ti, tj;           // first auxiliary row (A) and column (B) of the tile
  int m, n;             // rows and columns stored (<= 64, <= 128, even)
  int ktiles;           // nia_pad / 16
  int ldc;              // npad
  int diag;             // ti - tj: identity where col - row == diag
  int nw;               // frequencies (grid y)
  long long sC;         // doubles between the eps blocks of two frequencies
};
void launch_syrk_f64_tma(const F64SyrkItem* items, int n, int ny, cudaStream_t s);
cudaError_t prepare_syrk_f64_tma();

// chi0 on the tcgen05 cores: one upper tile of eps(iw) = 1 + M D_w M^T, 256 x 128 per pair of CTAs
// (digits) or 128 x 128 per CTA (tile_ctas), frequency = blockIdx.y (slab blockIdx.y).  The operand planes of M sqrt(D_w) are 3 to 7
// int8 digits (digit_gemm.cu; FP64: 7, RIGW_OZAKI(s): s) or two bf16 parts (syrk_bf16x3.cu; exps
// unused).
struct DigitItem {
  const void* maps;     // CUtensorMaps of the problem's planes (make_digit_tmaps)
  double* C;            // &eps[w0][0][0]
  int* err;
  const int* exps;      // digits, row exponents [w][ld]
  const unsigned long long* squares;   // digits: ProbDev::squares
  const int* negative;  // digits of FP64: not this kernel's problem when set (nullptr: always its)
  int rb_a, rb_b;       // 128-row blocks: output rows from 128 rb_a (two blocks of a pair, or one), columns from 128 rb_b
  int nrb, nkt;         // row blocks and k-tiles (64 transitions) of a slab
  int w0;               // frequency of slab 0
  int ld, nw;           // npad; frequencies covered
  long long sC;         // doubles between the eps blocks of two frequencies
};
// Update of finished rows on the digit products (digit_gemm.cu): C -= A^T B with A and B columns
// of [U | U^-T | U^-T M_sigma], digits of all rows above the tile, frequency = blockIdx.y.
struct UpdateItem {
  const void* maps;     // tensor maps of the problem's factor digits
  double* C;            // first row and column of the tile's region for j = 0
  int* err;
  const int* exps;      // [slab][group][128 nrb] column exponents
  int rb_a, rb_b;       // digit blocks of the output rows (two, of rows_a) and of the columns
  int nrb, nkt;         // digit blocks and k-tiles of a slab
  int nk, chunk;        // k-tiles summed; k-tiles per exponent group
  int first;            // first group that contributes (columns of U^-T are zero above their own)
  int ngroups;          // groups of a slab
  int slab, step;       // slab (frequency) for j = 0, and its increment
  int rows_a, ncol;     // row blocks present (1 or 2); columns stored
  int diag;             // 1: blocks below the diagonal (rb_b < row block) are not stored
  int ld, nw;
  long long sC;         // doubles between the regions of two j
};
// Digits of a group of finished rows: 128 columns of U, U^-T or U^-T M_sigma.
struct FactorSliceItem {
  const double* src;    // [rows][ld] for j = 0
  void* digits;
  int* exps;
  int ld, ncol, rows;
  int nrb, nkt, rb, kt; // digit blocks and k-tiles of a slab; block of the columns, first k-tile
  int ngroups, group;
  int slab, step, nw;
  long long s_src;
};
void launch_factor_slice(const FactorSliceItem* items, int n, int ny, cudaStream_t s);
void launch_digit_update(const UpdateItem* items, int n, int ny, cudaStream_t s);
void launch_digit_zero(const ProbDev* probs, const WorkItem* items, int n, cudaStream_t s);
void launch_digit_rowmax(const ProbDev* probs, const WorkItem* items, int n, cudaStream_t s);
// planes: digits per operand, 3 .. 7; ctas of a tile: 2, or 1 for up to six digits
void launch_digit_slice(int planes, const ProbDev* probs, const WorkItem* items, int n, cudaStream_t s);
void launch_digit_syrk(int planes, int ctas, const DigitItem* items, int n, int ny, cudaStream_t s);
void launch_split_bf16(const ProbDev* probs, const WorkItem* items, int n, cudaStream_t s);
void launch_split_syrk(const DigitItem* items, int n, int ny, cudaStream_t s);
cudaError_t prepare_digit_kernels();

// Host-side launchers of the DMMA tile engine (gemm_f64.cu).
// grid (n items) x (ny frequencies): CTAs with blockIdx.y >= item.nw return at once
void launch_dgemm_128x128(const GemmItem* items, int n, int ny, cudaStream_t s);
void launch_dgemm_64x128(const GemmItem* items, int n, int ny, cudaStream_t s);
void launch_dgemm_256x32(const GemmItem* items, int n, int ny, cudaStream_t s);   // narrow products
void launch_dgemm_128x64(const GemmItem* items, int n, int ny, cudaStream_t s);
void launch_dgemm_128x32(const GemmItem* items, int n, int ny, cudaStream_t s);   // 32-row warps
void launch_dgemm_64x32(const GemmItem* items, int n, int ny, cudaStream_t s);
cudaError_t prepare_dgemm_kernels();

}  // namespace rigw
