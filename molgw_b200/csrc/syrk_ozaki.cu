// Ozaki-sliced INT8 products of the AO->MO transform on the 5th-generation tensor cores
// (chi0 in RIGW_OZAKI modes: digit_gemm.cu).
//
//   row p of an operand is scaled by 2^-e_p, e_p the exponent of max_k |S_pk| (so |x| < 1):
//     x_pk = S_pk 2^-e_p = sum_{j=1..s} q_j(p,k) 2^-7j + r,  q_j integers in [-127, 127],
//   the base-128 digits of trunc(x 2^7s) (an exact 64-bit integer), with the sign of x.
//   (A B^T)_pq ~= 2^(e_p+f_q) sum_{d=2..s+1} 2^-7d L_d(p,q),   L_d = sum_{i+j=d} A_i B_j^T
//   (the products of level i+j > s+1 are dropped, as in the Ozaki scheme).
//
// L_d is an exact INT32 sum (tcgen05.mma kind::i8).  K is consumed in chunks of
// kOzChunk k-tiles (4096 entries): |L_d| <= s * 4096 * 127^2 < 2^31 on one
// chunk, so no sum can overflow; every (chunk, level) accumulator is drained
// into FP64 registers with its weight 2^-7d while the MMA warp fills another of
// the four TMEM accumulators.
//
// slice_rowmax_kernel, slice_kmajor_kernel: row exponents from the row maxima over K, and
//                      the s int8 slices K-major for TMA.
// syrk_ozaki_kernel:   one tile of A B^T per CTA; warp 0 issues
//                      TMA loads (one A and one B slice tile of 128 rows x 128
//                      entries per stage, 128-byte swizzle, 6 stages), warp 1
//                      issues the MMAs, warps 2..9 drain.  All waits are bounded.
#include "engine.cuh"
#include "tc_common.cuh"

namespace rigw {

// Base-128 digits of x (|x| < 1) truncated after s digits: X = trunc(x 2^(7s)) is
// exact in 64-bit integers (7s <= 49 bits), and digit k (k = 1..s) of |X|, with
// the sign of x, equals the k-th integer part taken by repeated x <- 128x - trunc(128x).
RIGW_DEVICE_INLINE long long ozaki_fixed(double x, int s) { return (long long)ldexp(x, 7 * s); }
RIGW_DEVICE_INLINE int ozaki_digit(long long X, int s, int k) {
  const long long a = X < 0 ? -X : X;
  const int d = int((a >> (7 * (s - k))) & 127);
  return X < 0 ? -d : d;
}

// ---------------------------------------------------------------------------
// General operands (the AO->MO products): 64 x 64 tiles through shared memory,
// read along the source's contiguous index.  Pass 1 takes the row maxima, pass 2
// the row exponents and the digits, written K-contiguous.
__global__ void __launch_bounds__(256) slice_rowmax_kernel(const SliceOp op) {
  __shared__ double tile[64][65];   // [row][k]
  __shared__ double part[4][64];
  const int k0 = blockIdx.x * 64, r0 = blockIdx.y * 64, z = blockIdx.z;
  const double* src = op.src + size_t(z) * op.zs_src;
  const bool rfast = op.rs == 1;
  const int tid = threadIdx.x;
  for (int idx = tid; idx < 64 * 64; idx += 256) {
    const int a = idx >> 6, b = idx & 63;
    const int rr = rfast ? b : a, kk = rfast ? a : b;
    const int r = r0 + rr, k = k0 + kk;
    tile[rr][kk] = (r < op.R && k < op.K) ? fabs(src[r * op.rs + k * op.ks]) : 0.0;
  }
  __syncthreads();
  const int rr = tid & 63, kq = tid >> 6;
  double m = 0.0;
#pragma unroll
  for (int kk = kq * 16; kk < kq * 16 + 16; ++kk) m = fmax(m, tile[rr][kk]);
  part[kq][rr] = m;
  __syncthreads();
  if (tid < 64) {
    m = fmax(fmax(part[0][tid], part[1][tid]), fmax(part[2][tid], part[3][tid]));
    if (m > 0.0) atomicMax(op.rmax + size_t(z) * op.Rpad + r0 + tid, (unsigned long long)__double_as_longlong(m));
  }
}

__global__ void __launch_bounds__(256) slice_kmajor_kernel(const SliceOp op) {
  __shared__ double tile[64][65];   // [row][k]
  __shared__ double rs[64];         // 2^-e_r
  const int k0 = blockIdx.x * 64, r0 = blockIdx.y * 64, z = blockIdx.z;
  const double* src = op.src + size_t(z) * op.zs_src;
  const bool rfast = op.rs == 1;
  const int tid = threadIdx.x, ns = op.slices;
  for (int idx = tid; idx < 64 * 64; idx += 256) {
    const int a = idx >> 6, b = idx & 63;
    const int rr = rfast ? b : a, kk = rfast ? a : b;
    const int r = r0 + rr, k = k0 + kk;
    tile[rr][kk] = (r < op.R && k < op.K) ? src[r * op.rs + k * op.ks] : 0.0;
  }
  if (tid < 64) {
    const size_t e_at = size_t(z) * op.Rpad + r0 + tid;
    const double m = __longlong_as_double((long long)op.rmax[e_at]);
    int e = 0;
    if (m > 0.0) frexp(m, &e);      // every |x| of the row is < 2^e
    rs[tid] = ldexp(1.0, -e);
    if (blockIdx.x == 0) op.exps[e_at] = e;
  }
  __syncthreads();
  int8_t* dst = reinterpret_cast<int8_t*>(op.dst);
  for (int idx = tid; idx < 64 * 32; idx += 256) {
    const int rr = idx >> 5, kp = (idx & 31) * 2;
    const long long X0 = ozaki_fixed(tile[rr][kp] * rs[rr], ns);
    const long long X1 = ozaki_fixed(tile[rr][kp + 1] * rs[rr], ns);
    for (int k = 1; k <= ns; ++k) {
      const size_t row = (size_t(z) * ns + k - 1) * op.Rpad + r0 + rr;
      *reinterpret_cast<char2*>(dst + row * op.Kpad + k0 + kp) =
          make_char2(char(ozaki_digit(X0, ns, k)), char(ozaki_digit(X1, ns, k)));
    }
  }
}

// ---------------------------------------------------------------------------
constexpr int kOzStages = 6;
constexpr int kOzTileBytes = 128 * 128;                 // 128 rows x 128 int8 transitions
constexpr int kOzStageBytes = 2 * kOzTileBytes;
constexpr size_t kOzSmemBytes = size_t(kOzStages) * kOzStageBytes + 1024 + 256;
constexpr int kOzChunk = 32;                            // k-tiles per exact INT32 accumulation
constexpr int kOzAcc = 4;                               // TMEM accumulators of 128 columns
constexpr int kOzThreads = 320;                         // warp 0 TMA, warp 1 MMA, warps 2..9 drain

__global__ void __launch_bounds__(kOzThreads, 1) syrk_ozaki_kernel(const TcItem* __restrict__ items) {
  const TcItem it = items[blockIdx.x];
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kOzStages * kOzStageBytes);
  uint64_t* empty = full + kOzStages;
  uint64_t* accf = empty + kOzStages;     // [kOzAcc] unit accumulated
  uint64_t* acce = accf + kOzAcc;         // [kOzAcc] unit drained
  uint32_t* tslot = reinterpret_cast<uint32_t*>(acce + kOzAcc);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto tile = [&](int s, int which) { return smem + s * kOzStageBytes + which * kOzTileBytes; };

  if (tid == 0) {
    for (int s = 0; s < kOzStages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < kOzAcc; ++b) {
      tc::mbar_init(&accf[b], 1);
      tc::mbar_init(&acce[b], 8);
    }
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(tslot, 128 * kOzAcc);
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;
  const int nk = it.ktiles;
  const int ns = it.slices;
  const int nchunks = (nk + kOzChunk - 1) / kOzChunk;
  // Work order (identical in the producer and the MMA issuer): chunk c, level
  // d = 2..ns+1, slice pair (i, d-i), k-tile of the chunk.  One unit = (c, d).

  if (tid == 0) {
    // ---- TMA producer
    tc::tmap_acquire(it.tmap);
    tc::tmap_acquire(it.tmap_b);
    int issued[kOzStages] = {0, 0, 0, 0, 0, 0};
    bool ok = true;
    int step = 0;
    for (int c = 0; c < nchunks && ok; ++c) {
      const int k0 = c * kOzChunk, k1 = min(nk, k0 + kOzChunk);
      for (int d = 2; d <= ns + 1 && ok; ++d)
        for (int i = max(1, d - ns); i <= min(ns, d - 1) && ok; ++i)
          for (int kt = k0; kt < k1; ++kt, ++step) {
            const int s = step % kOzStages;
            if (step >= kOzStages && !tc::mbar_wait(&empty[s], ((step / kOzStages) - 1) & 1)) {
              ok = false;
              break;
            }
            tc::mbar_arrive_expect_tx(&full[s], kOzStageBytes);
            tc::tma_load_2d(tile(s, 0), it.tmap, &full[s], kt * 128, it.row_a + (i - 1) * it.lo_off);
            tc::tma_load_2d(tile(s, 1), it.tmap_b, &full[s], kt * 128, it.row_b + (d - i - 1) * it.lo_off_b);
            ++issued[s];
          }
    }
    if (!ok) atomicOr(it.err, kErrTimeout);
    for (int s = 0; s < kOzStages; ++s)
      if (issued[s] > 0 && !tc::mbar_wait(&full[s], (issued[s] - 1) & 1)) atomicOr(it.err, kErrTimeout);
  } else if (tid == 32) {
    // ---- MMA issuer
    constexpr uint32_t idesc = tc::idesc_s8_s32(128, 128);
    bool ok = true;
    int step = 0, u = 0;
    for (int c = 0; c < nchunks && ok; ++c) {
      const int k0 = c * kOzChunk, k1 = min(nk, k0 + kOzChunk);
      for (int d = 2; d <= ns + 1 && ok; ++d, ++u) {
        const int b = u % kOzAcc;
        if (u >= kOzAcc && !tc::mbar_wait(&acce[b], ((u / kOzAcc) - 1) & 1)) {
          ok = false;
          break;
        }
        tc::tc_fence_after();
        const uint32_t dt = tmem + uint32_t(b * 128);
        bool first = true;
        for (int i = max(1, d - ns); i <= min(ns, d - 1) && ok; ++i)
          for (int kt = k0; kt < k1; ++kt, ++step) {
            const int s = step % kOzStages;
            if (!tc::mbar_wait(&full[s], (step / kOzStages) & 1)) {
              ok = false;
              break;
            }
            tc::tc_fence_after();
            const uint64_t ad = tc::desc_kmajor_sw128(tile(s, 0)), bd = tc::desc_kmajor_sw128(tile(s, 1));
#pragma unroll
            for (int sub = 0; sub < 4; ++sub) {
              const uint64_t o = uint64_t(sub * 2);   // 32 int8 = 32 bytes along K
              tc::mma_s8(dt, ad + o, bd + o, idesc, (first && sub == 0) ? 0u : 1u);
            }
            first = false;
            tc::mma_commit(&empty[s]);
          }
        if (ok) tc::mma_commit(&accf[b]);
      }
    }
    if (!ok) atomicOr(it.err, kErrTimeout);
  } else if (warp >= 2) {
    // ---- drain: every (chunk, level) accumulator into FP64 with weight 2^-7d
    const int quad = warp & 3;                 // TMEM lanes 32*quad .. 32*quad+31 (rows)
    const int half = (warp - 2) >> 2;          // columns 64*half .. 64*half+63
    const int row = quad * 32 + lane;
    double acc[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) acc[j] = 0.0;
    bool ok = true;
    int u = 0;
    for (int c = 0; c < nchunks && ok; ++c)
      for (int d = 2; d <= ns + 1; ++d, ++u) {
        const int b = u % kOzAcc;
        ok = __all_sync(0xffffffffu, tc::mbar_wait(&accf[b], (u / kOzAcc) & 1));
        if (!ok) break;
        tc::tc_fence_after();
        const double wd = ldexp(1.0, -7 * d);
        const uint32_t base = tmem + uint32_t(b * 128 + half * 64) + (uint32_t(quad * 32) << 16);
        uint32_t r[32];
        tc::tmem_ld_32x32(base, r);
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[j] += double(int(r[j])) * wd;
        tc::tmem_ld_32x32(base + 32, r);
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[32 + j] += double(int(r[j])) * wd;
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&acce[b]);
      }
    if (ok) {   // rows < mrows, columns < ncols
      if (row < it.mrows) {
        const int er = it.ea[row];
        double* dst = it.C + size_t(row) * it.ldc;
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          const int col = half * 64 + j;
          if (col < it.ncols) dst[col] = ldexp(acc[j], er + it.eb[col]);
        }
      }
    } else if (lane == 0) {
      atomicOr(it.err, kErrTimeout);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 128 * kOzAcc);
}

// ---------------------------------------------------------------------------
// Host side
void launch_slice_kmajor(const SliceOp& op, cudaStream_t s) {
  if (op.Rpad <= 0 || op.Kpad <= 0 || op.nz <= 0) return;
  cudaMemsetAsync(op.rmax, 0, size_t(op.nz) * op.Rpad * sizeof(unsigned long long), s);
  const dim3 grid(op.Kpad / 64, op.Rpad / 64, op.nz);
  slice_rowmax_kernel<<<grid, 256, 0, s>>>(op);
  slice_kmajor_kernel<<<grid, 256, 0, s>>>(op);
}
void launch_syrk_ozaki(const TcItem* items, int n, cudaStream_t s) {
  if (n > 0) syrk_ozaki_kernel<<<n, kOzThreads, kOzSmemBytes, s>>>(items);
}

cudaError_t prepare_ozaki_kernels() {
  return cudaFuncSetAttribute(syrk_ozaki_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kOzSmemBytes));
}

}  // namespace rigw
