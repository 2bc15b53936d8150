// chi0 from exact int8 digit products on the 5th-generation tensor cores: NS = 7 digits
// reach FP64 accuracy (RIGW_FP64 for all but the smallest problems), NS = s is RIGW_OZAKI(s).
//
//   eps(iw)[p][q] = delta_pq + sum_t S_pt S_qt,   S = M sqrt(D_w)
//
// Row p of S is scaled by a power of two to its largest entry and rounded once
// to an integer X of 8 NS - 1 bits; X is cut into NS balanced base-256 digits d_1 (most
// significant) .. d_NS, each an int8:  x = 2^(e_p - (8 NS - 1)) sum_i d_i 256^(NS - i).
//   (S S^T)_pq = 2^(e_p + e_q - 2 (8 NS - 1)) sum_{d=2}^{D} 256^(2 NS - d) L_d(p,q),
//   L_d = sum_{i+j=d} S_i S_j^T      (D = NS + 1, NS (NS + 1) / 2 digit products; D = 9, 34 of 49, for NS = 7)
// L_d is an exact INT32 sum (tcgen05.mma kind::i8) over chunks of kChunkTiles k-tiles: for
// NS = 7, |L_d| <= 7 * 128^2 * 16384 < 2^31.  The levels are joined in 64-bit integers,
// converted to FP64 once per chunk and summed in FP64.
//
// Error, NS = 7 (55-bit X), beside that of S in FP64 (2^-52 of each product): the entries are
// rounded to 2^-56 of their row's maximum, which puts a random error of 2^-56 max|S_p| |S_q| and its mirror image into the sum, at most
// 2^-55 sqrt(eps_pp eps_qq) whatever the spread of the entries and however long the sum,
// because a row maximum never exceeds the row's norm.  The products left out (i + j > 9) are
// digit products of zero mean with weight 2^-78 of the two row scales; K of them add up to
// 2^-64 sqrt(K) max|S_p| max|S_q|, which is less.  (Without level 9 they are 256 times that and
// the larger part: in rows that a few large entries dominate, 3 to 4 times the error of an
// FP64 sum.)  An FP64 sum rounds its running sum K times, about 2^-54 sqrt(K), beside M D_w.  Error against
// extended precision over that of FP64 sums (rms, relative to sqrt(eps_pp eps_qq)): normal
// entries 0.20 at 512 transitions, 0.05 at 4347; entries over three decades 0.23 and 0.05; three
// large entries a row 0.27 and 0.17.  (M D_w and M in place of S on both sides would not be
// bounded so: max|M_q| can exceed sqrt(eps_qq) by sqrt(max D / min D), 9 times the error of the
// FP64 sum for gaps over three decades and amplitudes that grow as their square roots, 512
// transitions.)
//
// 840 auxiliary functions, 4347 transitions, 32 frequencies: row maxima 0.04 ms, digits
// 0.16 ms, products 1.43 ms (3.5 Pop/s int8 over the executed tiles), against 4.25 ms on DMMA (23
// of 35 TF/s); 2000 / 25000 / 32: 0.37 + 2.19 + 35.4 ms against 111 ms.
// The operands are the same on both sides, so on the diagonal the products that are left out
// hold squares, whose mean is not zero.  If D + 1 is even, the first level left out has one, of
// digit (D + 1) / 2, which would lower eps_pp by 1e-9 for NS = 4 and by K 2^-66 max|S_p|^2 for
// NS = 7: digit_slice_kernel sums it per row, and it is added to the diagonal.  Otherwise the
// first square is 2^-8 below that level.
// A row that holds an infinity or a NaN gives NaN, as the FP64 sums did.  A negative D_w
// (inverted occupations) has no root: RIGW_FP64 then takes the DMMA kernel, which is launched
// behind these and returns at once unless digit_rowmax_kernel met one; in the sliced
// precisions the root is NaN and eps is reported as not positive definite.
//
// digit_rowmax_kernel: high words of max_t |S_pt| per frequency and row (integer maximum).
// digit_slice_kernel:  the digits of one frequency group, in the order in which the tensor
//   cores read them: [slab][row block of 128][k-tile of 64][digit][row group of 8][16-byte
//   k chunk][row][16 bytes], i.e. contiguous 8 x 16-byte core matrices, so that one TMA box
//   fetches all the digits of a tile.  One slab per frequency of the group.
// digit_syrk_kernel:   one 256 x 128 tile of eps(iw) per pair of CTAs (cta_group::2), or, for
//   small problems of up to six digits, one 128 x 128 tile per CTA.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <type_traits>

#include "engine.cuh"
#include "tc_common.cuh"

namespace rigw {

namespace {

constexpr int kNaNExp = 1 << 20;                 // row exponent of a row with a non-finite entry
constexpr int kDigThreads = 320;                 // warp 0 TMA, warp 1 MMA, warps 2..9 drain
constexpr int kChunkTiles = 256;                 // k-tiles (of 64) per exact INT32 accumulation
constexpr int kTileA = 128 * 64;                 // bytes of one digit of 128 rows

// CT: CTAs of a tile, a pair (256 x 128) or one (128 x 128; NS <= 6, whose slots leave room for two).
template <int NS, int CT = 2>
struct DigCfg {
  // last level summed: seven digits stand for FP64 and take one more than the NS + 1 whose weight
  // is that of the rounding of the entries
  static constexpr int kTop = NS == 7 ? NS + 2 : NS + 1;
  static constexpr int kLo = kTop - 1 < 4 ? kTop - 1 : 4;   // levels of the low pass: kTop + 1 - kLo .. kTop
  static constexpr int kHi = kTop - 1 - kLo;     // levels of the high pass: 2 .. kHi + 1 (digits 1 .. kHi)
  // the digit whose squares are added to the diagonal (0: none)
  static constexpr int kSquare = kTop % 2 ? (kTop + 1) / 2 : 0;
  static constexpr int kCtas = CT;
  static constexpr int kTileB = kTileA / kCtas;  // bytes of one digit of this CTA's rows of a B tile
  static constexpr int kSlot = NS * (kTileA + kTileB);
  static constexpr int kSlots = (216 * 1024) / kSlot;
  static constexpr int kPerHi = kHi > 0 ? NS / kHi : 1;   // k-tiles of the high pass per slot
  static constexpr size_t kSmem = size_t(kSlots) * kSlot + 1024 + 256;
};

// Exponent of a row from the high word of its largest |x|: |x| <= 0.996 * 2^e, so that the
// leading digit of rint(x 2^(8 NS - 1 - e)) is at most 127.
RIGW_DEVICE_INLINE int row_exponent(unsigned hi) {
  const int E = int(hi >> 20);
  if (E >= 2047) return kNaNExp;
  int e = (E == 0 ? 1 : E) - 1022;
  if (E > 0 && (hi & 0xfffffu) + 1u + 0x100000u > 2088763u) ++e;   // mantissa above 0.996
  return e < -960 ? -960 : e;
}

RIGW_DEVICE_INLINE double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }   // -1022 <= e <= 1023

// 2^e; NaN above 1023 (kNaNExp, also with a shift added), 2^-1022 at the least.
RIGW_DEVICE_INLINE double pow2_of(int e) {
  return e > 1023 ? __longlong_as_double(0x7ff8000000000000ll) : pow2(max(e, -1022));
}

}  // namespace

__global__ void __launch_bounds__(256) digit_zero_kernel(const ProbDev* __restrict__ probs,
                                                         const WorkItem* __restrict__ items) {
  const WorkItem wi = items[blockIdx.x];
  const ProbDev& p = probs[wi.prob];
  const int n = p.nomega * p.npad;
  if (p.negative && wi.a == 0 && threadIdx.x == 0) *p.negative = 0;
  for (int k = threadIdx.x; k < 4096; k += 256)
    if (wi.a + k < n) {
      p.dmax[wi.a + k] = 0u;
      p.squares[wi.a + k] = 0;
    }
}

// item: (prob, t0, row block): split_t transitions from t0, 128 rows, every frequency.
// Thread (row, half) keeps 32 entries of its row in registers and walks the frequencies:
// one FP64 product and one integer maximum per entry and frequency.
__global__ void __launch_bounds__(256) digit_rowmax_kernel(const ProbDev* __restrict__ probs,
                                                           const WorkItem* __restrict__ items) {
  const WorkItem wi = items[blockIdx.x];
  const ProbDev& p = probs[wi.prob];
  constexpr int kWb = 16;
  __shared__ double sd[kWb][64];
  const int tid = threadIdx.x, row = tid & 127, half = tid >> 7;
  const int r = wi.b * 128 + row;
  const int tend = min(p.nia_pad, wi.a + p.split_t);
  for (int t0 = wi.a; t0 < tend; t0 += 64) {
    double v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = p.mp[size_t(t0 + half * 32 + i) * p.npad + r];
    for (int wb = 0; wb < p.nomega; wb += kWb) {
      const int nwb = min(kWb, p.nomega - wb);
      __syncthreads();
      for (int i = tid; i < nwb * 64; i += 256) {
        const double d = p.dscale[size_t(wb + (i >> 6)) * p.nia_pad + t0 + (i & 63)];
        if (d < 0.0 && p.negative) *p.negative = 1;   // any thread: the same value
        sd[i >> 6][i & 63] = sqrt(d);
      }
      __syncthreads();
      for (int w = 0; w < nwb; ++w) {
        unsigned m = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i)
          m = max(m, unsigned(__double2hiint(v[i] * sd[w][half * 32 + i])) & 0x7fffffffu);
        if (m) atomicMax(p.dmax + size_t(wb + w) * p.npad + r, m);
      }
    }
  }
}

namespace {

// 4 x 4 byte transpose: o[b] = byte b of w0, w1, w2, w3.
RIGW_DEVICE_INLINE void bytes4(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, uint32_t (&o)[4]) {
  const uint32_t a = __byte_perm(w0, w1, 0x5140), b = __byte_perm(w2, w3, 0x5140);
  const uint32_t c = __byte_perm(w0, w1, 0x7362), d = __byte_perm(w2, w3, 0x7362);
  o[0] = __byte_perm(a, b, 0x5410);
  o[1] = __byte_perm(a, b, 0x7632);
  o[2] = __byte_perm(c, d, 0x5410);
  o[3] = __byte_perm(c, d, 0x7632);
}

// The NS digits of 16 consecutive transitions of one row: X = rint(v scale), a carry-in of
// 128 in every byte but the leading one makes the digits balanced, and 16 bytes per digit
// go to core-matrix row `dst` (digit planes kTileA bytes apart).  Returns the sum of the squares
// of digit kSquare.
template <int NS>
RIGW_DEVICE_INLINE int write_digits(const double (&v)[16], double scale, int8_t* dst) {
  constexpr uint64_t kBias = NS >= 8 ? 0x0080808080808080ull : (0x8080808080808080ull & ((1ull << (8 * (NS - 1))) - 1));
  uint32_t out[NS][4];
#pragma unroll
  for (int g = 0; g < 4; ++g) {
    uint32_t lo[4], hi[4], o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint64_t y = (uint64_t(__double2ll_rn(v[4 * g + i] * scale)) + kBias) ^ kBias;
      lo[i] = uint32_t(y);
      hi[i] = uint32_t(y >> 32);
    }
    bytes4(lo[0], lo[1], lo[2], lo[3], o);
#pragma unroll
    for (int b = 0; b < 4 && b < NS; ++b) out[NS - 1 - b][g] = o[b];
    if (NS > 4) {
      bytes4(hi[0], hi[1], hi[2], hi[3], o);
#pragma unroll
      for (int b = 4; b < NS; ++b) out[NS - 1 - b][g] = o[b - 4];
    }
  }
#pragma unroll
  for (int s = 0; s < NS; ++s)
    *reinterpret_cast<uint4*>(dst + size_t(s) * kTileA) = make_uint4(out[s][0], out[s][1], out[s][2], out[s][3]);
  int sq = 0;
  if constexpr (DigCfg<NS>::kSquare > 0) {
    const auto& m = out[DigCfg<NS>::kSquare - 1];
#pragma unroll
    for (int g = 0; g < 4; ++g) sq = __dp4a(int(m[g]), int(m[g]), sq);
  }
  return sq;
}

// Byte offset of (slab, row block, k-tile, digit 1, row, 16-byte chunk kc) in the digit array.
RIGW_DEVICE_INLINE size_t digit_offset(int slab, int nrb, int rb, int nkt, int kt, int ns, int row, int kc) {
  return (((size_t(slab) * nrb + rb) * nkt + kt) * ns) * kTileA + size_t(row >> 3) * 512 + kc * 128 + (row & 7) * 16;
}

}  // namespace

// item: (prob, k-tile, row block, w0): the frequencies w0 .. w0 + wgroup - 1 into slabs 0 ...
// A warp writes 32 rows of one 16-byte chunk: four full lines
// per digit.  Memory bound: NS bytes written per entry and frequency (840 auxiliary
// functions, 32 frequencies: 0.87 GB).
template <int NS>
__global__ void __launch_bounds__(256) digit_slice_kernel(const ProbDev* __restrict__ probs,
                                                          const WorkItem* __restrict__ items) {
  const WorkItem wi = items[blockIdx.x];
  const ProbDev& p = probs[wi.prob];
  if (p.negative && *p.negative) return;   // left to DMMA
  constexpr int kWb = 16;
  __shared__ double sd[kWb][64];
  const int tid = threadIdx.x, row = tid & 127, half = tid >> 7;
  const int kt = wi.a, rb = wi.b, r = rb * 128 + row, t0 = kt * 64;
  const int nrb = p.npad / 128, nkt = p.nia_pad / 64;
  int8_t* dig = reinterpret_cast<int8_t*>(p.xs);
  double v[2][16];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int i = 0; i < 16; ++i) v[c][i] = p.mp[size_t(t0 + (half * 2 + c) * 16 + i) * p.npad + r];
  const int w0 = wi.c, w1 = min(p.nomega, w0 + p.wgroup);
  for (int wb = w0; wb < w1; wb += kWb) {
    const int nwb = min(kWb, w1 - wb);
    __syncthreads();
    for (int i = tid; i < nwb * 64; i += 256)
      sd[i >> 6][i & 63] = sqrt(p.dscale[size_t(wb + (i >> 6)) * p.nia_pad + t0 + (i & 63)]);
    __syncthreads();
    for (int w = 0; w < nwb; ++w) {
      const int e = row_exponent(p.dmax[size_t(wb + w) * p.npad + r]);
      if (kt == 0 && half == 0) p.xexp[size_t(wb + w) * p.npad + r] = e;
      const double sc = pow2(8 * NS - 1 - (e == kNaNExp ? 0 : e));
      int sq = 0;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        double x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = v[c][i] * sd[w][(half * 2 + c) * 16 + i];
        sq += write_digits<NS>(x, sc, dig + digit_offset(wb - w0 + w, nrb, rb, nkt, kt, NS, row, half * 2 + c));
      }
      if (DigCfg<NS>::kSquare > 0) atomicAdd(p.squares + size_t(wb + w) * p.npad + r, (unsigned long long)(sq));
    }
  }
}

// One 256 x 128 tile per CTA pair: rank r holds A rows 128 r .. and B rows 64 r .. of the
// tile and accumulates output rows 128 r ...  A slot of the ring holds every digit of one
// k-tile of 64 transitions (84 KB per CTA for NS = 7, two slots; five slots of 32 transitions
// measured 2% slower), so each digit tile that is loaded feeds all the products it appears
// in; tcgen05 reads 96 bytes of shared memory per clock and CTA and
// TMA writes 30, below the 128 that shared memory delivers (a 128 x 128 tile of one CTA
// would read 128 and write 45).  TMEM holds four 128-column accumulators, so the levels go
// in two passes over a chunk: the four lowest levels (24 of the 34 products for NS = 7), and
// the rest from the leading digits alone, as many k-tiles per slot as fit.
template <int NS, int CT, class Item>
__device__ __forceinline__ void digit_product(const Item& it, const int jw) {
  using Cfg = DigCfg<NS, CT>;
  constexpr int kTileB = Cfg::kTileB;
  constexpr bool kPair = Cfg::kCtas == 2;
  constexpr bool kUpdate = std::is_same<Item, UpdateItem>::value;
  extern __shared__ uint8_t dig_smem_raw[];
  uint8_t* smem =
      reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dig_smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + Cfg::kSlots * Cfg::kSlot);   // used in rank 0
  uint64_t* empty = full + Cfg::kSlots;     // slot read by the MMAs (both ranks)
  uint64_t* accf = empty + Cfg::kSlots;     // pass accumulated (both ranks)
  uint64_t* acce = accf + 1;                // pass drained by the 16 warps of the pair (rank 0)
  uint32_t* tslot = reinterpret_cast<uint32_t*>(acce + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = kPair ? int(tc::cluster_rank()) : 0;
  if (tid == 0) {
    for (int s = 0; s < Cfg::kSlots; ++s) {
      tc::mbar_init(&full[s], 1);
      tc::mbar_init(&empty[s], 1);
    }
    tc::mbar_init(accf, 1);
    tc::mbar_init(acce, 8 * Cfg::kCtas);
    tc::fence_mbar_init();
  }
  if (warp == 0) {
    if constexpr (kPair) tc::tmem_alloc_pair(tslot, 512);
    else tc::tmem_alloc(tslot, 512);
  }
  __syncthreads();
  if constexpr (kPair) tc::cluster_sync();        // the peer's barriers are initialised
  tc::tc_fence_after();
  const uint32_t tmem = *tslot;
  int nk, chunk, slab;                // k-tiles summed, k-tiles per chunk, slab of both operands
  int c0 = 0;                         // first chunk
  if constexpr (kUpdate) {
    nk = it.nk;
    chunk = it.chunk;
    c0 = it.first;
    slab = it.slab + jw * it.step;
  } else {
    nk = it.nkt;
    chunk = kChunkTiles;
    slab = jw;
  }
  const int nchunks = (nk + chunk - 1) / chunk;
  constexpr int kPasses = Cfg::kHi > 0 ? 2 : 1;
  // k-tiles of a slot in pass q (0: low levels, 1: high levels)
  auto per_slot = [](int q) { return q == 0 ? 1 : Cfg::kPerHi; };
  auto slot = [&](int s) { return smem + s * Cfg::kSlot; };

  if (tid == 0) {
    // ---- TMA producer of this CTA; rank 0's full barrier counts the bytes of both
    const uint8_t* maps = static_cast<const uint8_t*>(it.maps);
    for (int m = 0; m < (kPasses > 1 ? 4 : 2); ++m) tc::tmap_acquire(maps + 128 * m);
    const int rowA = (slab * it.nrb + it.rb_a + rank) * it.nkt;
    const int rowB = (slab * it.nrb + it.rb_b) * it.nkt;
    uint32_t issued = 0;
    bool ok = true;
    for (int c = c0; c < nchunks && ok; ++c)
      for (int q = 0; q < kPasses && ok; ++q) {
        const int k1 = min(nk, (c + 1) * chunk), ps = per_slot(q);
        const int nd = q == 0 ? NS : Cfg::kHi;             // digits loaded
        for (int k0 = c * chunk; k0 < k1; k0 += ps, ++issued) {
          const int s = int(issued % Cfg::kSlots);
          if (issued >= uint32_t(Cfg::kSlots) &&
              !tc::mbar_wait(&empty[s], ((issued / Cfg::kSlots) - 1) & 1)) {
            ok = false;
            break;
          }
          const int nt = min(ps, k1 - k0);
          if (rank == 0) tc::mbar_arrive_expect_tx(&full[s], uint32_t(Cfg::kCtas * nt * nd * (kTileA + kTileB)));
          const uint32_t bar = kPair ? tc::mapa(&full[s], 0) : 0;
          for (int t = 0; t < nt; ++t) {
            uint8_t* d = slot(s) + t * nd * (kTileA + kTileB);
            if constexpr (kPair) {
              tc::tma_load_3d_pair(d, maps + 256 * q, bar, 0, 0, (rowA + k0 + t) * NS);
              tc::tma_load_3d_pair(d + nd * kTileA, maps + 256 * q + 128, bar, 0, 32 * rank, (rowB + k0 + t) * NS);
            } else {
              tc::tma_load_3d(d, maps + 256 * q, &full[s], 0, 0, (rowA + k0 + t) * NS);
              tc::tma_load_3d(d + nd * kTileA, maps + 256 * q, &full[s], 0, 0, (rowB + k0 + t) * NS);
            }
          }
        }
      }
    if (!ok) atomicOr(it.err, kErrTimeout);
    // copies still in flight on a timeout land before the CTA leaves (bounded wait)
    if (rank == 0) {
      for (uint32_t s = 0; s < uint32_t(Cfg::kSlots) && s < issued; ++s) {
        const uint32_t last = issued - 1 - (issued - 1 - s) % Cfg::kSlots;
        if (!tc::mbar_wait(&full[s], (last / Cfg::kSlots) & 1)) atomicOr(it.err, kErrTimeout);
      }
    } else if (!ok) {
      const uint64_t t0 = tc::global_ns();
      while (tc::global_ns() - t0 < 1000000ull) {
      }
    }
  } else if (tid == 32 && rank == 0) {
    // ---- MMA issuer of the pair
    constexpr uint32_t idesc = tc::idesc_s8_s32(128 * Cfg::kCtas, 128);
    bool ok = true;
    uint32_t step = 0;
    int pass = 0;
    for (int c = c0; c < nchunks && ok; ++c)
#pragma unroll
      for (int q = 0; q < kPasses; ++q) {
        if (!ok) break;
        if (pass > 0 && !tc::mbar_wait(acce, (pass - 1) & 1)) {
          ok = false;
          break;
        }
        ++pass;
        tc::tc_fence_after();
        const int k1 = min(nk, (c + 1) * chunk), ps = per_slot(q);
        constexpr int kBytesLo = NS * (kTileA + kTileB);
        uint32_t first = 0u;
        for (int k0 = c * chunk; k0 < k1; k0 += ps, ++step) {
          const int s = int(step % Cfg::kSlots);
          if (!tc::mbar_wait(&full[s], (step / Cfg::kSlots) & 1)) {
            ok = false;
            break;
          }
          tc::tc_fence_after();
          const int nt = min(ps, k1 - k0);
          for (int t = 0; t < nt; ++t) {
            const int nd = q == 0 ? NS : Cfg::kHi;
            const uint8_t* base = slot(s) + (q == 0 ? 0 : t * nd * (kTileA + kTileB));
            static_assert(kBytesLo == Cfg::kSlot, "one k-tile per slot in the low pass");
            const uint64_t ad = tc::desc_kmajor_cores(base, 512);
            const uint64_t bd = tc::desc_kmajor_cores(base + nd * kTileA, 512);
            const int nl = q == 0 ? Cfg::kLo : Cfg::kHi;
            const int d0 = q == 0 ? Cfg::kTop + 1 - Cfg::kLo : 2;
#pragma unroll
            for (int a = 0; a < nl; ++a) {
              const int d = d0 + a;
              const uint32_t dt = tmem + uint32_t(a * 128);
              bool fresh = true;
#pragma unroll
              for (int i = 1; i <= NS; ++i) {
                const int j = d - i;
                if (j < 1 || j > NS) continue;
#pragma unroll
                for (int sub = 0; sub < 2; ++sub) {
                  // 32 int8 along K = two core matrices = 256 bytes
                  const uint64_t ai = ad + uint64_t(((i - 1) * kTileA + sub * 256) >> 4);
                  const uint64_t bj = bd + uint64_t(((j - 1) * kTileB + sub * 256) >> 4);
                  const uint32_t keep = (fresh && sub == 0) ? first : 1u;
                  if constexpr (kPair) tc::mma_s8_pair(dt, ai, bj, idesc, keep);
                  else tc::mma_s8(dt, ai, bj, idesc, keep);
                }
                fresh = false;
              }
            }
            first = 1u;
          }
          if constexpr (kPair) tc::mma_commit_pair(&empty[s]);
          else tc::mma_commit(&empty[s]);
        }
        if (ok) {
          if constexpr (kPair) tc::mma_commit_pair(accf);
          else tc::mma_commit(accf);
        }
      }
    if (!ok) atomicOr(it.err, kErrTimeout);
  } else if (warp >= 2) {
    // ---- drain: join the levels of a pass in 64-bit integers, add to FP64 registers
    const int quad = warp & 3;                 // TMEM lanes 32 quad .. (rows)
    const int half = (warp - 2) >> 2;          // columns 64 half ..
    const uint32_t done = kPair ? tc::mapa(acce, 0) : 0;
    // weight of the lowest level of unit-scaled operands
    constexpr int kShift = 8 * (2 * NS - Cfg::kTop) - 2 * (8 * NS - 1);
    double acc[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) acc[j] = 0.0;
    bool ok = true;
    int pass = 0;
    for (int c = c0; c < nchunks && ok; ++c)
#pragma unroll
      for (int q = 0; q < kPasses; ++q) {
        if (!ok) break;
        ok = __all_sync(0xffffffffu, tc::mbar_wait(accf, pass & 1));
        if (!ok) break;
        ++pass;
        tc::tc_fence_after();
        constexpr int kLoL = Cfg::kLo, kHiL = Cfg::kHi;
        const double wq = q == 0 ? 1.0 : double(1ull << (8 * kLoL));
        // update: every chunk has row and column exponents of its own
        double wr = wq * pow2(kShift);   // a power of two, at least 2^-1030
        const int* ecol = nullptr;
        if constexpr (kUpdate) {
          const int* e = it.exps + (size_t(slab) * it.ngroups + c) * it.nrb * 128;
          wr *= pow2_of(e[min(it.rb_a + rank, it.nrb - 1) * 128 + quad * 32 + lane]);
          ecol = e + it.rb_b * 128 + half * 64;
        }
#pragma unroll
        for (int cb = 0; cb < 8; ++cb) {
          const uint32_t base = tmem + uint32_t(half * 64 + cb * 8) + (uint32_t(quad * 32) << 16);
          uint32_t r[4][8];
          const int nl = q == 0 ? kLoL : kHiL;
#pragma unroll
          for (int a = 0; a < 4; ++a)
            if (a < nl) tc::tmem_ld_32x8(base + uint32_t(a * 128), r[a]);
          tc::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            long long x = int(r[0][j]);
#pragma unroll
            for (int a = 1; a < 4; ++a)
              if (a < nl) x = x * 256 + int(r[a][j]);
            if constexpr (kUpdate) acc[cb * 8 + j] += double(x) * (wr * pow2_of(ecol[cb * 8 + j]));
            else acc[cb * 8 + j] += double(x) * wq;
          }
        }
        tc::tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if constexpr (kPair) tc::mbar_arrive_cluster(done);
          else tc::mbar_arrive(acce);
        }
      }
    if (!ok) {
      if (lane == 0) atomicOr(it.err, kErrTimeout);
    } else if constexpr (kUpdate) {
      if (rank < it.rows_a && !(it.diag && it.rb_b < it.rb_a + rank)) {
        double* dst = it.C + jw * it.sC + size_t(rank * 128 + quad * 32 + lane) * it.ld + half * 64;
#pragma unroll
        for (int j = 0; j < 64; j += 2) {
          if (half * 64 + j >= it.ncol) break;     // an even number of columns
          double2 v = *reinterpret_cast<const double2*>(dst + j);
          v.x -= acc[j];
          v.y -= acc[j + 1];
          *reinterpret_cast<double2*>(dst + j) = v;
        }
      }
    } else {
      const int rb = it.rb_a + rank, cb = it.rb_b;
      if (rb < it.nrb && rb <= cb) {               // blocks below the diagonal are not stored
        const int row = rb * 128 + quad * 32 + lane, col0 = cb * 128 + half * 64;
        const int* exps = it.exps + size_t(it.w0 + jw) * it.ld;
        const int er = exps[row];
        // what the diagonal element of this row gets beside its products: the squares of the level
        // below the lowest and the identity (read once: per column it cost 20 us in a diagonal tile)
        double diag = 0.0;
        if (Cfg::kSquare > 0 && rb == cb)
          diag = ldexp(double(it.squares[size_t(it.w0 + jw) * it.ld + row]), 2 * er + kShift - 8);
        double* dst = it.C + jw * it.sC + size_t(row) * it.ld + col0;
#pragma unroll
        for (int j = 0; j < 64; j += 2) {
          double v[2];
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int ec = exps[col0 + j + u];
            v[u] = (er == kNaNExp || ec == kNaNExp) ? __longlong_as_double(0x7ff8000000000000ll)
                                                     : ldexp(acc[j + u], er + ec + kShift);
            if (col0 + j + u == row) v[u] = v[u] + diag + 1.0;
          }
          *reinterpret_cast<double2*>(dst + j) = make_double2(v[0], v[1]);
        }
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if constexpr (kPair) tc::cluster_sync();        // no CTA leaves while its peer may still reach its memory
  if (warp == 0) {
    __syncwarp();
    if constexpr (kPair) tc::tmem_dealloc_pair(tmem, 512);
    else tc::tmem_dealloc(tmem, 512);
  }
}

// Grid x: the items times CT, in clusters of that size.
template <int NS, int CT>
__global__ void __cluster_dims__(CT, 1, 1) __launch_bounds__(kDigThreads, 1)
    digit_syrk_kernel(const DigitItem* __restrict__ items) {
  const DigitItem it = items[blockIdx.x / CT];
  // both CTAs of the pair, before any barrier or TMEM use
  if (int(blockIdx.y) >= it.nw || (it.negative && *it.negative)) return;
  digit_product<NS, CT>(it, blockIdx.y);
}

// C -= A^T B for the rows of one panel group, A and B columns of the finished rows above it
// (the factorization of eps and its fused solves).  The columns' digits are scaled group of
// rows by group of rows, so a chunk of the sum is one group and is joined with its own weights:
// U's entries far above the diagonal are small, and one scale for a whole column would have to
// cover its largest entry.  DMMA did these updates at 20 TF/s (64 x 128 tiles, K = 256 at a
// time, every trailing tile read and written once per group); here each tile is written once
// in all, with K of all rows above (2000 auxiliary functions, 32 frequencies: stage 15.6 -> 10.3 ms).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kDigThreads, 1)
    digit_update_kernel(const UpdateItem* __restrict__ items) {
  const UpdateItem it = items[blockIdx.x >> 1];
  if (int(blockIdx.y) >= it.nw) return;
  digit_product<kFp64Digits, 2>(it, blockIdx.y);
}

// One block of 128 columns of a group of finished rows: column maxima, then the digits, both
// passes over the same rows (the second one from L2).  Thread (column, half).
__global__ void __launch_bounds__(256) factor_slice_kernel(const FactorSliceItem* __restrict__ items) {
  const FactorSliceItem it = items[blockIdx.x];
  const int jw = blockIdx.y;
  if (jw >= it.nw) return;
  __shared__ unsigned part[2][128];
  const int tid = threadIdx.x, col = tid & 127, half = tid >> 7;
  const double* src = it.src + jw * it.s_src + col;
  const bool live = col < it.ncol;
  unsigned m = 0;
  if (live) {
#pragma unroll 8
    for (int r = half; r < it.rows; r += 2)
      m = max(m, unsigned(__double2hiint(src[size_t(r) * it.ld])) & 0x7fffffffu);
  }
  part[half][col] = m;
  __syncthreads();
  const int e = row_exponent(max(part[0][col], part[1][col]));
  const int slab = it.slab + jw * it.step;
  if (half == 0) it.exps[((size_t(slab) * it.ngroups + it.group) * it.nrb + it.rb) * 128 + col] = e;
  const double sc = pow2(8 * kFp64Digits - 1 - (e == kNaNExp ? 0 : e));
  int8_t* dig = static_cast<int8_t*>(it.digits);
  for (int kt = 0; kt < it.rows / 64; ++kt)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int kc = half * 2 + c;
      double v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = live ? src[size_t(kt * 64 + kc * 16 + i) * it.ld] : 0.0;
      write_digits<kFp64Digits>(v, sc,
                                dig + digit_offset(slab, it.nrb, it.rb, it.nkt, it.kt + kt, kFp64Digits, col, kc));
    }
}

// ---------------------------------------------------------------------------
// Host side
namespace {
PFN_cuTensorMapEncodeTiled_v12000 g_encode_dig = nullptr;

template <int NS, int CT>
cudaError_t prepare_ns() {
  return cudaFuncSetAttribute(digit_syrk_kernel<NS, CT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              int(DigCfg<NS, CT>::kSmem));
}
template <int NS, int CT>
void syrk_ns(const DigitItem* items, int n, int ny, cudaStream_t s) {
  digit_syrk_kernel<NS, CT><<<dim3(CT * n, ny), kDigThreads, DigCfg<NS, CT>::kSmem, s>>>(items);
}
}  // namespace

// Four maps (512 bytes) of `planes` operand planes (slabs x row blocks x k-tiles x ns) of
// `cores` core matrices of 128 bytes (64: int8 digits, 128: bf16): all planes of an A tile and
// of half a B tile, then the leading digits of the high pass.
Status make_digit_tmaps(void* host_maps, const void* digits, long long planes, int ns, int cores) {
  if (!g_encode_dig) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qr;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr) != cudaSuccess ||
        qr != cudaDriverEntryPointSuccess || !fn) {
      cudaGetLastError();
      return Status::fail(RIGW_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
    }
    g_encode_dig = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  CUtensorMap* maps = reinterpret_cast<CUtensorMap*>(host_maps);
  const int nhi = ns == 7 ? 4 : (ns > 4 ? ns - 4 : 1);   // DigCfg::kHi
  for (int m = 0; m < 4; ++m) {
    cuuint64_t dims[3] = {128, cuuint64_t(cores), cuuint64_t(planes)};
    cuuint64_t strides[2] = {128, cuuint64_t(128 * cores)};
    cuuint32_t box[3] = {128, cuuint32_t(m & 1 ? cores / 2 : cores), cuuint32_t(m < 2 ? ns : nhi)};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult e = g_encode_dig(&maps[m], CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(digits), dims, strides, box,
                              estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (e != CUDA_SUCCESS) return Status::fail(RIGW_ERR_CUDA, "cuTensorMapEncodeTiled (digits) failed (%d)", int(e));
  }
  return Status::ok();
}

void launch_digit_zero(const ProbDev* probs, const WorkItem* items, int n, cudaStream_t s) {
  if (n > 0) digit_zero_kernel<<<n, 256, 0, s>>>(probs, items);
}
void launch_digit_rowmax(const ProbDev* probs, const WorkItem* items, int n, cudaStream_t s) {
  if (n > 0) digit_rowmax_kernel<<<n, 256, 0, s>>>(probs, items);
}
void launch_digit_slice(int planes, const ProbDev* probs, const WorkItem* items, int n, cudaStream_t s) {
  if (n <= 0) return;
  switch (planes) {
    case 3: digit_slice_kernel<3><<<n, 256, 0, s>>>(probs, items); break;
    case 4: digit_slice_kernel<4><<<n, 256, 0, s>>>(probs, items); break;
    case 5: digit_slice_kernel<5><<<n, 256, 0, s>>>(probs, items); break;
    case 6: digit_slice_kernel<6><<<n, 256, 0, s>>>(probs, items); break;
    default: digit_slice_kernel<7><<<n, 256, 0, s>>>(probs, items); break;
  }
}
void launch_factor_slice(const FactorSliceItem* items, int n, int ny, cudaStream_t s) {
  if (n > 0 && ny > 0) factor_slice_kernel<<<dim3(n, ny), 256, 0, s>>>(items);
}
void launch_digit_update(const UpdateItem* items, int n, int ny, cudaStream_t s) {
  if (n > 0 && ny > 0)
    digit_update_kernel<<<dim3(2 * n, ny), kDigThreads, DigCfg<kFp64Digits>::kSmem, s>>>(items);
}
// ctas: of a tile (see DigCfg); 1 for planes <= 6 only
void launch_digit_syrk(int planes, int ctas, const DigitItem* items, int n, int ny, cudaStream_t s) {
  if (n <= 0 || ny <= 0) return;
  switch (planes * 10 + ctas) {
    case 31: syrk_ns<3, 1>(items, n, ny, s); break;
    case 32: syrk_ns<3, 2>(items, n, ny, s); break;
    case 41: syrk_ns<4, 1>(items, n, ny, s); break;
    case 42: syrk_ns<4, 2>(items, n, ny, s); break;
    case 51: syrk_ns<5, 1>(items, n, ny, s); break;
    case 52: syrk_ns<5, 2>(items, n, ny, s); break;
    case 61: syrk_ns<6, 1>(items, n, ny, s); break;
    case 62: syrk_ns<6, 2>(items, n, ny, s); break;
    default: syrk_ns<7, 2>(items, n, ny, s); break;
  }
}
cudaError_t prepare_digit_kernels() {
  for (cudaError_t e : {prepare_ns<3, 1>(), prepare_ns<3, 2>(), prepare_ns<4, 1>(), prepare_ns<4, 2>(),
                        prepare_ns<5, 1>(), prepare_ns<5, 2>(), prepare_ns<6, 1>(), prepare_ns<6, 2>(),
                        prepare_ns<7, 2>()})
    if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(digit_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              int(DigCfg<kFp64Digits>::kSmem));
}

}  // namespace rigw
