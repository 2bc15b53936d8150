// Split-precision products on the 5th-generation tensor cores.
//
//   eps(iw) = 1 + S S^T,   S = M diag(sqrt(D_w)) = S_hi + S_lo  (bf16 hi/lo split)
//   S S^T  ~=  S_hi S_hi^T + S_hi S_lo^T + S_lo S_hi^T     (fp32 accumulation in TMEM)
//
// split_bf16_kernel: scales the packed FP64 tensor by sqrt(D_w(t)) for every frequency of a
//   group and writes the hi/lo pair in the order in which the tensor cores read it
//   (8 x 16-byte core matrices, as digit_gemm.cu).
// split_syrk_kernel: one 128 x 128 upper tile of eps(iw) per CTA.
// split_kmajor_kernel, syrk_bf16x3_kernel: the general products of the AO->MO transform,
//   one 128 x 128 tile per CTA from K-major operands (128-byte swizzle).
// All mbarrier waits are bounded.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "engine.cuh"
#include "tc_common.cuh"

namespace rigw {

constexpr int kTcStages = 3;
constexpr int kTcTileBytes = 128 * 64 * 2;
constexpr int kTcStageBytes = 4 * kTcTileBytes;
constexpr size_t kTcSmemBytes = size_t(kTcStages) * kTcStageBytes + 1024 + 256;

// A bf16 value, as the bits of the float it is, in FP64.  Integer arithmetic: a conversion
// instruction runs at a quarter of the FP64 rate, and three per entry bounded the kernel.  Exact
// for normal values; below 2^-126 it is off by less than 2^-125, and a NaN or an infinity has
// already gone into the high part.
RIGW_DEVICE_INLINE double widen(uint32_t u) {
  return __hiloint2double(int((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), 0);
}

// item: (prob, k-tile, row block, w0): frequencies w0 .. w0 + wgroup - 1 into slabs 0 ...
// Thread (row, half) keeps 32 entries of its row for all frequencies; a warp writes 32 rows
// of one 16-byte chunk, four full lines.
__global__ void __launch_bounds__(256) split_bf16_kernel(const ProbDev* __restrict__ probs,
                                                         const WorkItem* __restrict__ items) {
  const WorkItem wi = items[blockIdx.x];
  const ProbDev& p = probs[wi.prob];
  constexpr int kWb = 16;
  constexpr int kPlane = 128 * 128;     // bytes of hi or lo of 128 rows x 64 transitions
  __shared__ double sd[kWb][64];
  const int tid = threadIdx.x, row = tid & 127, half = tid >> 7;
  const int kt = wi.a, rb = wi.b, r = rb * 128 + row, t0 = kt * 64 + half * 32;
  const int nrb = p.npad / 128, nkt = p.nia_pad / 64;
  double v[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = p.mp[size_t(t0 + i) * p.npad + r];
  uint8_t* out = static_cast<uint8_t*>(p.xs) + size_t(row >> 3) * 1024 + (row & 7) * 16 + half * 512;
  auto write = [&](const double* d, int slab) {   // d: factors of the 32 transitions
    uint8_t* dst = out + (((size_t(slab) * nrb + rb) * nkt + kt) * 2) * kPlane;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint32_t hi[4], lo[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int k = c * 8 + 2 * i;
        const double x0 = v[k] * d[k], x1 = v[k + 1] * d[k + 1];
        const __nv_bfloat162 h = __floats2bfloat162_rn(float(x0), float(x1));
        hi[i] = *reinterpret_cast<const uint32_t*>(&h);
        // the low part from the FP64 remainder (through FP32, whose rounding is 2^-16 of its own)
        const __nv_bfloat162 l = __floats2bfloat162_rn(float(x0 - widen(hi[i] << 16)),
                                                       float(x1 - widen(hi[i] & 0xffff0000u)));
        lo[i] = *reinterpret_cast<const uint32_t*>(&l);
      }
      *reinterpret_cast<uint4*>(dst + c * 128) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
      *reinterpret_cast<uint4*>(dst + kPlane + c * 128) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
  };
  const int w0 = wi.c, w1 = min(p.nomega, w0 + p.wgroup);
  for (int wb = w0; wb < w1; wb += kWb) {
    const int nwb = min(kWb, w1 - wb);
    __syncthreads();
    for (int i = tid; i < nwb * 64; i += 256)
      sd[i >> 6][i & 63] = sqrt(p.dscale[size_t(wb + (i >> 6)) * p.nia_pad + kt * 64 + (i & 63)]);
    __syncthreads();
    for (int w = 0; w < nwb; ++w) write(&sd[w][half * 32], wb - w0 + w);
  }
}

// General operand split: 64 (rows) x 64 (K) tiles through shared memory, read
// along the source's contiguous index and written K-contiguous.
__global__ void __launch_bounds__(256) split_kmajor_kernel(const SplitOp op) {
  __shared__ double tile[64][65];   // [row][k]
  const int k0 = blockIdx.x * 64, r0 = blockIdx.y * 64, z = blockIdx.z;
  const double* src = op.src + size_t(z) * op.zs_src;
  __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(op.dst) + size_t(z) * op.zs_dst;
  const bool rfast = op.rs == 1;
  for (int idx = threadIdx.x; idx < 64 * 64; idx += 256) {
    const int a = idx >> 6, b = idx & 63;
    const int rr = rfast ? b : a, kk = rfast ? a : b;
    const int r = r0 + rr, k = k0 + kk;
    tile[rr][kk] = (r < op.R && k < op.K) ? src[r * op.rs + k * op.ks] : 0.0;
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < 64 * 64; idx += 256) {
    const int rr = idx >> 6, kk = idx & 63;
    const double v = tile[rr][kk];
    const __nv_bfloat16 h = __double2bfloat16(v);
    const __nv_bfloat16 l = __double2bfloat16(v - double(__bfloat162float(h)));
    const size_t o = size_t(r0 + rr) * op.Kpad + k0 + kk;
    dst[o] = h;
    dst[o + size_t(op.Rpad) * op.Kpad] = l;
  }
}

// K is consumed in chunks of 512 transitions that accumulate in fp32 in one of two TMEM
// accumulators (128 columns each); eight drain warps per CTA add a finished chunk to FP64
// registers while the MMA warp fills the other, so the fp32 accumulation length is bounded
// whatever the number of transitions.
//
// One 128 x 128 tile per CTA.  What bounds the products is the traffic into shared memory: 64 KB
// per k-tile of 64 transitions from L2, two boxes of both parts of an operand each, in the order in
// which the tensor cores read them.  A 256 x 128 tile per CTA pair (cta_group::2) loads a quarter
// less, but computes rows beyond the last block and blocks below the diagonal, and its two CTAs
// wait for each other; the row-major form with four 128-byte-swizzled boxes per k-tile needs more
// instructions and transactions.  chi0 stage, row-major / pairs / this (ms): 64 molecules of 128
// auxiliary functions 0.301 / 0.381 / 0.242, 32 of 300 1.11 / 1.28 / 0.97, 8 of 700 2.36 / 2.41 /
// 2.08; one of 768 0.348 / 0.387 / 0.321, 840 0.502 / 0.490 / 0.452, 1700 5.39 / 5.73 / 4.98, 2000
// 9.74 / 9.14 / 8.97, 4000 (48 frequencies) 249 / 246 / 239.
constexpr int kSpPlane = 128 * 128;                        // hi or lo of 128 rows, 64 transitions
constexpr int kSpSlot = 4 * kSpPlane;                      // 64 KB
constexpr int kSpSlots = 3;
constexpr int kSpChunk = 8;                                // k-tiles per fp32 accumulation
constexpr int kSpThreads = 320;                            // warp 0 TMA, warp 1 MMA, warps 2..9 drain
constexpr size_t kSpSmem = size_t(kSpSlots) * kSpSlot + 1024 + 256;

__global__ void __launch_bounds__(kSpThreads, 1) split_syrk_kernel(const DigitItem* __restrict__ items) {
  const DigitItem it = items[blockIdx.x];
  const int jw = blockIdx.y;
  if (jw >= it.nw) return;   // before any barrier or TMEM use
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kSpSlots * kSpSlot);
  uint64_t* empty = full + kSpSlots;        // slot read by the MMAs
  uint64_t* accf = empty + kSpSlots;        // [2] chunk accumulated
  uint64_t* acce = accf + 2;                // [2] chunk drained by the 8 warps
  uint32_t* tslot = reinterpret_cast<uint32_t*>(acce + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int s = 0; s < kSpSlots; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&accf[b], 1);
      tc::mbar_init(&acce[b], 8);
    }
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(tslot, 256);
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;
  const int nk = it.nkt;
  const int nchunks = (nk + kSpChunk - 1) / kSpChunk;

  if (tid == 0) {
    // ---- TMA producer
    tc::tmap_acquire(it.maps);
    const int rowA = (jw * it.nrb + it.rb_a) * nk;
    const int rowB = (jw * it.nrb + it.rb_b) * nk;
    int issued = 0;
    bool ok = true;
    for (int kt = 0; kt < nk; ++kt, ++issued) {
      const int s = kt % kSpSlots;
      if (kt >= kSpSlots && !tc::mbar_wait(&empty[s], ((kt / kSpSlots) - 1) & 1)) {
        ok = false;
        break;
      }
      tc::mbar_arrive_expect_tx(&full[s], kSpSlot);
      uint8_t* d = smem + s * kSpSlot;
      tc::tma_load_3d(d, it.maps, &full[s], 0, 0, (rowA + kt) * 2);
      tc::tma_load_3d(d + 2 * kSpPlane, it.maps, &full[s], 0, 0, (rowB + kt) * 2);
    }
    if (!ok) atomicOr(it.err, kErrTimeout);
    // copies still in flight on a timeout land before the CTA leaves (bounded wait)
    for (int s = 0; s < kSpSlots && s < issued; ++s)
      if (!tc::mbar_wait(&full[s], (((issued - 1 - s) / kSpSlots)) & 1)) atomicOr(it.err, kErrTimeout);
  } else if (tid == 32) {
    // ---- MMA issuer
    constexpr uint32_t idesc = tc::idesc_bf16_f32(128, 128);
    bool ok = true;
    for (int kt = 0; kt < nk && ok; ++kt) {
      const int c = kt / kSpChunk, b = c & 1;
      const bool first = (kt % kSpChunk) == 0;
      if (first && c >= 2 && !tc::mbar_wait(&acce[b], ((c >> 1) - 1) & 1)) {
        ok = false;
        break;
      }
      const int s = kt % kSpSlots;
      if (!tc::mbar_wait(&full[s], (kt / kSpSlots) & 1)) {
        ok = false;
        break;
      }
      tc::tc_fence_after();
      const uint32_t d = tmem + uint32_t(b * 128);
      const uint8_t* base = smem + s * kSpSlot;
      const uint64_t ah = tc::desc_kmajor_cores(base, 1024), al = tc::desc_kmajor_cores(base + kSpPlane, 1024);
      const uint64_t bh = tc::desc_kmajor_cores(base + 2 * kSpPlane, 1024);
      const uint64_t bl = tc::desc_kmajor_cores(base + 3 * kSpPlane, 1024);
#pragma unroll
      for (int sub = 0; sub < 4; ++sub) {
        const uint64_t o = uint64_t(sub * 16);   // 16 bf16 along K = two core matrices = 256 bytes
        tc::mma_bf16(d, ah + o, bh + o, idesc, (first && sub == 0) ? 0u : 1u);
        tc::mma_bf16(d, ah + o, bl + o, idesc, 1u);
        tc::mma_bf16(d, al + o, bh + o, idesc, 1u);
      }
      tc::mma_commit(&empty[s]);
      if ((kt % kSpChunk) == kSpChunk - 1 || kt == nk - 1) tc::mma_commit(&accf[b]);
    }
    if (!ok) atomicOr(it.err, kErrTimeout);
  } else if (warp >= 2) {
    // ---- drain each chunk into FP64 registers, then store the tile
    const int quad = warp & 3;                 // TMEM lanes 32 quad .. (rows)
    const int half = (warp - 2) >> 2;          // columns 64 half ..
    double acc[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) acc[j] = 0.0;
    bool ok = true;
    for (int c = 0; c < nchunks; ++c) {
      const int b = c & 1;
      ok = __all_sync(0xffffffffu, tc::mbar_wait(&accf[b], (c >> 1) & 1));
      if (!ok) break;
      tc::tc_fence_after();
      const uint32_t base = tmem + uint32_t(b * 128 + half * 64) + (uint32_t(quad * 32) << 16);
#pragma unroll
      for (int cb = 0; cb < 8; ++cb) {
        uint32_t r[8];
        tc::tmem_ld_32x8(base + cb * 8, r);
        tc::tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[cb * 8 + j] += double(__uint_as_float(r[j]));
      }
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acce[b]);
    }
    const int rb = it.rb_a, cb = it.rb_b;
    if (!ok) {
      if (lane == 0) atomicOr(it.err, kErrTimeout);
    } else {
      const int row = rb * 128 + quad * 32 + lane, col0 = cb * 128 + half * 64;
      double* dst = it.C + jw * it.sC + size_t(row) * it.ld + col0;
#pragma unroll
      for (int j = 0; j < 64; j += 2) {
        double v0 = acc[j], v1 = acc[j + 1];
        if (col0 + j == row) v0 += 1.0;
        if (col0 + j + 1 == row) v1 += 1.0;
        *reinterpret_cast<double2*>(dst + j) = make_double2(v0, v1);
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    __syncwarp();
    tc::tmem_dealloc(tmem, 256);
  }
}

// The general product of the AO->MO transform: the same chunks, one 128 x 128 tile per CTA.
constexpr int kTcChunk = 8;
constexpr int kTcThreads = 320;    // warp 0 TMA, warp 1 MMA, warps 2..9 epilogue

__global__ void __launch_bounds__(kTcThreads, 1) syrk_bf16x3_kernel(const TcItem* __restrict__ items) {
  const TcItem it = items[blockIdx.x];
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kTcStages * kTcStageBytes);
  uint64_t* empty = full + kTcStages;
  uint64_t* accf = empty + kTcStages;     // [2] chunk accumulated
  uint64_t* acce = accf + 2;              // [2] chunk drained
  uint32_t* tslot = reinterpret_cast<uint32_t*>(acce + 2);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto tile = [&](int s, int which) { return smem + s * kTcStageBytes + which * kTcTileBytes; };

  if (tid == 0) {
    for (int s = 0; s < kTcStages; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&accf[b], 1);
      tc::mbar_init(&acce[b], 8);
    }
    tc::fence_mbar_init();
  }
  if (warp == 0) tc::tmem_alloc(tslot, 256);
  __syncthreads();
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;
  const int nk = it.ktiles;
  const int nchunks = (nk + kTcChunk - 1) / kTcChunk;

  if (tid == 0) {
    // ---- TMA producer
    tc::tmap_acquire(it.tmap);
    tc::tmap_acquire(it.tmap_b);
    int issued[kTcStages] = {0, 0, 0};
    bool ok = true;
    for (int kt = 0; kt < nk && ok; ++kt) {
      const int s = kt % kTcStages;
      if (kt >= kTcStages && !tc::mbar_wait(&empty[s], ((kt / kTcStages) - 1) & 1)) {
        ok = false;
        break;
      }
      tc::mbar_arrive_expect_tx(&full[s], kTcStageBytes);
      const int k0 = kt * 64;
      tc::tma_load_2d(tile(s, 0), it.tmap, &full[s], k0, it.row_a);
      tc::tma_load_2d(tile(s, 1), it.tmap, &full[s], k0, it.row_a + it.lo_off);
      tc::tma_load_2d(tile(s, 2), it.tmap_b, &full[s], k0, it.row_b);
      tc::tma_load_2d(tile(s, 3), it.tmap_b, &full[s], k0, it.row_b + it.lo_off_b);
      ++issued[s];
    }
    if (!ok) atomicOr(it.err, kErrTimeout);
    for (int s = 0; s < kTcStages; ++s)
      if (issued[s] > 0 && !tc::mbar_wait(&full[s], (issued[s] - 1) & 1)) atomicOr(it.err, kErrTimeout);
  } else if (tid == 32) {
    // ---- MMA issuer
    constexpr uint32_t idesc = tc::idesc_bf16_f32(128, 128);
    bool ok = true;
    for (int kt = 0; kt < nk && ok; ++kt) {
      const int c = kt / kTcChunk, b = c & 1;
      const bool first = (kt % kTcChunk) == 0;
      if (first && c >= 2 && !tc::mbar_wait(&acce[b], ((c >> 1) - 1) & 1)) {
        ok = false;
        break;
      }
      const int s = kt % kTcStages;
      if (!tc::mbar_wait(&full[s], (kt / kTcStages) & 1)) {
        ok = false;
        break;
      }
      tc::tc_fence_after();
      const uint32_t d = tmem + uint32_t(b * 128);
      const uint64_t ah = tc::desc_kmajor_sw128(tile(s, 0)), al = tc::desc_kmajor_sw128(tile(s, 1));
      const uint64_t bh = tc::desc_kmajor_sw128(tile(s, 2)), bl = tc::desc_kmajor_sw128(tile(s, 3));
#pragma unroll
      for (int sub = 0; sub < 4; ++sub) {
        const uint64_t o = uint64_t(sub * 2);   // 16 bf16 = 32 bytes along K
        tc::mma_bf16(d, ah + o, bh + o, idesc, (first && sub == 0) ? 0u : 1u);
        tc::mma_bf16(d, ah + o, bl + o, idesc, 1u);
        tc::mma_bf16(d, al + o, bh + o, idesc, 1u);
      }
      tc::mma_commit(&empty[s]);
      if ((kt % kTcChunk) == kTcChunk - 1 || kt == nk - 1) tc::mma_commit(&accf[b]);
    }
    if (!ok) atomicOr(it.err, kErrTimeout);
  } else if (warp >= 2) {
    // ---- epilogue: drain each chunk into FP64 registers, then store the tile
    const int quad = warp & 3;                 // TMEM lanes 32*quad .. 32*quad+31 (rows)
    const int half = (warp - 2) >> 2;          // columns 64*half .. 64*half+63
    const int row = quad * 32 + lane;
    double acc[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) acc[j] = 0.0;
    bool ok = true;
    for (int c = 0; c < nchunks; ++c) {
      const int b = c & 1;
      ok = __all_sync(0xffffffffu, tc::mbar_wait(&accf[b], (c >> 1) & 1));
      if (!ok) break;
      tc::tc_fence_after();
      const uint32_t base = tmem + uint32_t(b * 128 + half * 64) + (uint32_t(quad * 32) << 16);
      uint32_t r[32];
      tc::tmem_ld_32x32(base, r);
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] += double(__uint_as_float(r[j]));
      tc::tmem_ld_32x32(base + 32, r);
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[32 + j] += double(__uint_as_float(r[j]));
      tc::tc_fence_before();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acce[b]);
    }
    if (ok) {   // rows < mrows, columns < ncols
      if (row < it.mrows) {
        double* dst = it.C + size_t(row) * it.ldc;
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if (half * 64 + j < it.ncols) dst[half * 64 + j] = acc[j];
      }
    } else if (lane == 0) {
      atomicOr(it.err, kErrTimeout);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------
// Host side
namespace {
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
}

bool bf16x3_available() {
  if (g_encode) return true;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !fn) {
    cudaGetLastError();
    return false;
  }
  g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  return true;
}

// Row-major [rows][kpad] tensor read in boxes of 128 rows x 128 bytes (128-byte swizzle).
static Status make_kmajor_tmap(void* host_map, CUtensorMapDataType type, int esize, const void* base, int kpad,
                               long long rows) {
  if (!bf16x3_available()) return Status::fail(RIGW_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
  CUtensorMap* m = reinterpret_cast<CUtensorMap*>(host_map);
  cuuint64_t dims[2] = {cuuint64_t(kpad), cuuint64_t(rows)};
  cuuint64_t strides[1] = {cuuint64_t(kpad) * esize};
  cuuint32_t box[2] = {cuuint32_t(128 / esize), 128};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode(m, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return Status::fail(RIGW_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", int(r));
  return Status::ok();
}

Status make_split_tmap(void* host_map, const void* xs, int kpad, long long rows) {
  return make_kmajor_tmap(host_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, xs, kpad, rows);
}

Status make_ozaki_tmap(void* host_map, const void* xq, int kpad, long long rows) {
  return make_kmajor_tmap(host_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, xq, kpad, rows);
}

void launch_split_bf16(const ProbDev* probs, const WorkItem* items, int n, cudaStream_t s) {
  if (n > 0) split_bf16_kernel<<<n, 256, 0, s>>>(probs, items);
}

void launch_split_syrk(const DigitItem* items, int n, int ny, cudaStream_t s) {
  if (n > 0 && ny > 0) split_syrk_kernel<<<dim3(n, ny), kSpThreads, kSpSmem, s>>>(items);
}

void launch_split_kmajor(const SplitOp& op, cudaStream_t s) {
  if (op.Rpad > 0 && op.Kpad > 0 && op.nz > 0)
    split_kmajor_kernel<<<dim3(op.Kpad / 64, op.Rpad / 64, op.nz), 256, 0, s>>>(op);
}

void launch_syrk_bf16x3(const TcItem* items, int n, cudaStream_t s) {
  if (n > 0) syrk_bf16x3_kernel<<<n, kTcThreads, kTcSmemBytes, s>>>(items);
}

cudaError_t prepare_tc_kernels() {
  cudaError_t e = cudaFuncSetAttribute(split_syrk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSpSmem));
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(syrk_bf16x3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kTcSmemBytes));
}

}  // namespace rigw
