// Trailing update of the FP64 LU on the tensor cores (tcgen05, sm_100a).
//
//     A22 <- A22 - L21 * U12        (complex FP64, inner dimension K = 128 per panel)
//
// B200's FP64 pipe multiplies at 30 TFLOP/s (measured); its INT8 tensor pipe is
// two orders of magnitude wider and exact. So each operand is split into
// integer slices (the error-free splitting of Ozaki, Ogita, Oishi and Rump):
// row r of L21 (column c of U12) gets one power-of-two scale 2^e above its
// largest component over the panel, every component becomes the 55-bit integer
// V = rint(x 2^(54 - e)), and V its seven balanced base-256 digits
//     V = sum_t d_t 256^t,  d_t in [-128, 127].
// Slice i holds the digits of weight 256^(6 - i). A product of two slices is
// exact in INT32 over K = 64 complex (2 * 64 * 7 * 2^14 < 2^31), products of
// equal i + j share an accumulator (a diagonal), and the diagonals are summed in
// FP64 with their powers of 256.
//
// Diagonals i + j <= 7 are kept (34 slice products). What is dropped is below
// 2^-58 of the row's and column's maxima, what the 55-bit rounding loses below
// 2^-55 of one maximum. Measured on the influence matrices of six hulls (300 to
// 780 panels, deep and finite depth, 80-bit reference): the factors' and the
// solutions' errors are those of an FP64 multiply-add chain to within 2%
// (e.g. 3.5e-16 and 3.6e-16); with the 28 products of i + j <= 6 the solutions'
// error is up to 45% larger, so the eighth diagonal stays.
//
// The complex product is real: A as [Ar | Ai] along k, B as the planes
// [-Bi; Br; Bi] of 64 columns each, of which Ar multiplies (Br, Bi) and Ai
// multiplies (-Bi, Br): two neighbouring planes each, so B needs three planes
// instead of four.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "linalg.cuh"
#include "tc_gemm.cuh"

namespace nb200 {

constexpr int OZ_S = 7;                          // slices per operand
constexpr int OZ_D = 8;                          // diagonals kept: i + j <= 7
constexpr int OZ_M = 128;                        // rows per tile
constexpr int OZ_N = 64;                         // complex columns per tile (128 accumulator columns: Re, Im)
constexpr int OZ_KC = 64;                        // complex k per chunk
constexpr int OZ_NCH = LU_OUTER / OZ_KC;         // chunks per panel
constexpr int OZ_A = OZ_M * 2 * OZ_KC;           // 16 KB: one slice of an A chunk
constexpr int OZ_PLANE = OZ_N * OZ_KC;           // 4 KB: one plane of a B slice
constexpr int OZ_B = 3 * OZ_PLANE;               // 12 KB: one slice of a B chunk
constexpr int OZ_ASBO = 2 * OZ_KC * 8;           // bytes between 8-row groups of an A slice
constexpr int OZ_BSBO = OZ_KC * 8;               // and of a B plane
constexpr int OZ_SLOT = OZ_A + OZ_B;             // 28 KB: slice i of both operands
constexpr int OZ_SLOTS = 8;                      // the seven slices of a chunk and one ahead
constexpr int OZ_ACC = 4;                        // accumulators of 128 tensor-memory columns
constexpr int OZ_THREADS = 320;                  // producer, MMA issuer, eight epilogue warps
constexpr int OZ_EPI = 256;
constexpr int OZ_SMEM = OZ_SLOTS * OZ_SLOT + 256;
constexpr int OZ_EMIN = -250;                    // smallest scale exponent (rows and columns below it are round-off)
// Trailing entries of a batch (over its systems) from which an update takes this
// path; below it the FP64 pipe's one launch is as fast as the images and the
// update, which then cover few SMs. LU in ms, FP64 pipe against this path: 10
// systems of 420 panels (0.9 M entries) 0.74 / 0.82, 4 of 894 (2.3 M) 1.37 / 1.45,
// 2 of 1,430 (3.4 M) 2.23 / 2.26, 20 of 588 (4.2 M) 1.47 / 1.47, 1 of 2,380 (5.1 M)
// 4.19 / 3.99, 4 of 1,430 (6.8 M) 3.06 / 2.80, 20 of 2,380 (101 M) 37.8 / 22.2.
constexpr double OZ_MIN_ENTRIES = 4.2e6;
// slices in the order a chunk needs them: the first diagonal (i + j = 7) starts
// from the middle, slice 0 is not in it
constexpr unsigned OZ_ORDER = 0x0162543u;        // nibble p: the p-th slice loaded

// Operand images and scales of two panels (the update of one panel may be
// merged into the next one's): per system and set, ceil(n / 128) row tiles and
// 2 ceil(n / 128) column tiles of OZ_NCH chunks of OZ_S slices; scales one per
// row, then one per column.
struct OzWork {
  unsigned char* a = nullptr;
  unsigned char* b = nullptr;
  double* sc = nullptr;
  size_t have_a = 0, have_b = 0, have_sc = 0;
  int tiles = 0;   // row tiles per system of the current batch (set by ensure)
  int nsys = 0;
  size_t bytes() const { return have_a + have_b + have_sc; }
  void release() {
    cudaFree(a);
    cudaFree(b);
    cudaFree(sc);
    a = b = nullptr;
    sc = nullptr;
    have_a = have_b = have_sc = 0;
  }
  ~OzWork() { release(); }
  cudaError_t ensure(int ns, int n, bool headroom = false) {
    tiles = (n + OZ_M - 1) / OZ_M;
    nsys = ns;
    const size_t t = 2 * (size_t)ns * tiles;
    cudaError_t e = grow_alloc(reinterpret_cast<void**>(&a), &have_a, t * OZ_NCH * OZ_S * OZ_A, headroom);
    if (e) return e;
    e = grow_alloc(reinterpret_cast<void**>(&b), &have_b, t * 2 * OZ_NCH * OZ_S * OZ_B, headroom);
    if (e) return e;
    return grow_alloc(reinterpret_cast<void**>(&sc), &have_sc, t * 2 * OZ_M * sizeof(double), headroom);
  }
};
inline size_t oz_bytes_per_system(size_t n) {
  const size_t t = 2 * ((n + OZ_M - 1) / OZ_M);
  return t * (OZ_NCH * OZ_S * (size_t)(OZ_A + 2 * OZ_B) + 2 * OZ_M * sizeof(double));
}

// The images of one panel as the kernels take them (bases of the launch's
// first system): strides are per system.
struct OzSet {
  unsigned char* a = nullptr;
  unsigned char* b = nullptr;
  double* ra = nullptr;   // row scales
  double* cb = nullptr;   // column scales
};
struct OzStride {
  long long a, b, s;
};
inline OzStride oz_stride(const OzWork& w) {
  return OzStride{(long long)w.tiles * OZ_NCH * OZ_S * OZ_A, (long long)w.tiles * 2 * OZ_NCH * OZ_S * OZ_B,
                  (long long)w.tiles * OZ_M};
}
inline OzSet oz_set(const OzWork& w, int set, int s0) {
  const OzStride st = oz_stride(w);
  const long long q = (long long)set * w.nsys + s0;
  OzSet r;
  r.a = w.a + q * st.a;
  r.b = w.b + q * st.b;
  r.ra = w.sc + q * st.s;
  r.cb = w.sc + ((long long)2 * w.nsys + q) * st.s;
  return r;
}

// 16 components scaled by 2^(54 - e): their digits, slice by slice, as 16-byte
// rows out(i, uint4). V + 0x0080..80 has the digits offset by 128 as its bytes,
// so the digits are those bytes with the top bit flipped.
template <class Out>
__device__ __forceinline__ void oz_digits(const double* x, double scale, bool neg, Out out) {
  uint32_t w[OZ_S][4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      long long v = __double2ll_rn(x[4 * q + j] * scale);
      if (neg) v = -v;
      const unsigned long long u =
          ((unsigned long long)(v + 0x0080808080808080ll)) ^ 0x0080808080808080ull;
      lo[j] = (uint32_t)u;
      hi[j] = (uint32_t)(u >> 32);
    }
    // byte t of the four values, in order, is the word of slice 6 - t
    auto quad = [](const uint32_t* v, uint32_t& b0, uint32_t& b1, uint32_t& b2, uint32_t& b3) {
      const uint32_t p = __byte_perm(v[0], v[1], 0x5140), q2 = __byte_perm(v[2], v[3], 0x5140);
      const uint32_t r = __byte_perm(v[0], v[1], 0x7362), s = __byte_perm(v[2], v[3], 0x7362);
      b0 = __byte_perm(p, q2, 0x5410);
      b1 = __byte_perm(p, q2, 0x7632);
      b2 = __byte_perm(r, s, 0x5410);
      b3 = __byte_perm(r, s, 0x7632);
    };
    uint32_t top;
    quad(lo, w[6][q], w[5][q], w[4][q], w[3][q]);
    quad(hi, w[2][q], w[1][q], w[0][q], top);
  }
#pragma unroll
  for (int i = 0; i < OZ_S; ++i) out(i, make_uint4(w[i][0], w[i][1], w[i][2], w[i][3]));
}

// exponent field of the largest magnitude so far; NaN and infinities sort above
// every finite value
__device__ __forceinline__ unsigned oz_mag(double x, unsigned m) {
  return max(m, (unsigned)__double2hiint(x) & 0x7fffffffu);
}
__device__ __forceinline__ int oz_exponent(unsigned mag) { return max((int)(mag >> 20) - 1022, OZ_EMIN); }
__device__ __forceinline__ double oz_pow2(int e) { return __hiloint2double((1023 + e) << 20, 0); }
// what one row's digits are worth in the result: the kept diagonals weigh
// 256^7 .. 1 in units of 256^5 of both operands, 2^20 of each. A row with a
// NaN or an infinity makes every result of the row NaN.
__device__ __forceinline__ double oz_scale(unsigned mag, int e) {
  return mag >= 0x7ff00000u ? __longlong_as_double(0x7ff8000000000000ll) : oz_pow2(e - 34);
}

// Images of the panel [k0, k0 + 128): L21 = A[r1:n, k0:r1] and U12 = A[k0:r1,
// r1:n], r1 = k0 + 128. Blocks [0, na): 32 rows of L21, thread = (row, 16 k);
// the others: 32 columns of U12, thread = (column, 16 k). Reads 16 B and writes
// 14 B (L21) or 21 B (U12) per entry, bound by HBM and the FP64 -> INT64
// conversions; one pass over the operands, which stay in registers between the
// maximum and the digits.
constexpr int OZP_THREADS = 256;
__global__ void __launch_bounds__(OZP_THREADS) oz_prep_kernel(Batch b, int k0, OzSet s, OzStride st, int na) {
  __shared__ unsigned red[8][32];
  const int n = b.order(blockIdx.z), r1 = k0 + LU_OUTER, rest = n - r1;
  if (rest <= 0) return;
  const int padded = (rest + OZ_M - 1) / OZ_M * OZ_M;
  const double2* A = b.sys(blockIdx.z);
  const bool isA = (int)blockIdx.x < na;
  const int base = (isA ? blockIdx.x : blockIdx.x - na) * 32;
  if (base >= padded) return;
  const int t = threadIdx.x;
  const int g = isA ? t >> 5 : t & 7;                // k-group of 16
  const int rr = base + (isA ? t & 31 : t >> 3);     // row or column within the trailing block
  const int kb = k0 + 16 * g;
  double re[16], im[16];
  unsigned mag = 0;
  const bool in = r1 + rr < n;
  const double2* p = isA ? A + (r1 + rr) + (long long)n * kb : A + kb + (long long)n * (r1 + rr);
  const long long step = isA ? n : 1;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const double2 v = in ? p[step * j] : make_double2(0., 0.);
    re[j] = v.x;
    im[j] = v.y;
    mag = oz_mag(v.y, oz_mag(v.x, mag));
  }
  if (isA) {
    red[g][t & 31] = mag;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) mag = max(mag, red[q][t & 31]);
  } else {
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) mag = max(mag, __shfl_xor_sync(0xffffffffu, mag, o));
  }
  const int e = oz_exponent(mag);
  const double sc = oz_pow2(54 - e);
  const int ch = g / (OZ_KC / 16), kg = g % (OZ_KC / 16);
  if (isA) {
    if (g == 0) s.ra[blockIdx.z * st.s + rr] = oz_scale(mag, e);
    const int row = rr % OZ_M;
    unsigned char* img = s.a + blockIdx.z * st.a + ((long long)(rr / OZ_M) * OZ_NCH + ch) * OZ_S * OZ_A +
                         (row & 7) * 16 + (row >> 3) * OZ_ASBO + kg * 128;
    oz_digits(re, sc, false, [&](int i, uint4 v) { *reinterpret_cast<uint4*>(img + i * OZ_A) = v; });
    oz_digits(im, sc, false, [&](int i, uint4 v) { *reinterpret_cast<uint4*>(img + i * OZ_A + (OZ_KC / 16) * 128) = v; });
  } else {
    if (g == 0) s.cb[blockIdx.z * st.s + rr] = oz_scale(mag, e);
    const int col = rr % OZ_N;
    unsigned char* img = s.b + blockIdx.z * st.b + ((long long)(rr / OZ_N) * OZ_NCH + ch) * OZ_S * OZ_B +
                         (col & 7) * 16 + (col >> 3) * OZ_BSBO + kg * 128;
    oz_digits(im, sc, true, [&](int i, uint4 v) { *reinterpret_cast<uint4*>(img + i * OZ_B) = v; });
    oz_digits(re, sc, false, [&](int i, uint4 v) { *reinterpret_cast<uint4*>(img + i * OZ_B + OZ_PLANE) = v; });
    oz_digits(im, sc, false, [&](int i, uint4 v) { *reinterpret_cast<uint4*>(img + i * OZ_B + 2 * OZ_PLANE) = v; });
  }
}

// bounded wait that lets the hardware suspend the thread: at most 2^20 tries of
// about a microsecond each
__device__ __forceinline__ bool mbar_wait_suspend(uint32_t bar, uint32_t parity) {
  for (int i = 0; i < (1 << 20); ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(1000u)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// instruction descriptor of kind::i8: S32 accumulator, signed 8-bit A and B,
// K-major, M = 128, N = 128
constexpr uint32_t OZ_IDESC =
    (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)((2 * OZ_N) >> 3) << 17) | ((uint32_t)(OZ_M >> 4) << 24);

__device__ __forceinline__ void oz_mma(uint32_t tmem, uint64_t da, uint64_t db, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
      "l"(da), "l"(db), "r"(OZ_IDESC), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t* v) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(addr));
}

// The update of a rectangle of tiles (row tiles [ti0, ti0 + nti), column tiles
// [tj0, tj0 + ntc) of 128 x 64 complex) of every system, one persistent CTA per
// SM walking tile t, t + grid, ...:
//   warp 0 (one thread)  loads slice i of A and B (28 KB) into one of eight
//                        slots; the slots free up as the diagonals go down;
//   warp 1 (one thread)  issues the MMAs of a chunk diagonal by diagonal, i + j
//                        = 7 first, then 6 .. 0 (slice s is done with diagonal
//                        s, so its slot takes the next chunk's slice while the
//                        diagonals below still run), each into one of four
//                        128-column accumulators;
//   warps 2-9            add a finished diagonal to the tile's FP64 sums (64 per
//                        thread, in registers; warp w the TMEM lanes 32 (w % 4)
//                        .. and half (w - 2) / 4 of the columns) and, after the
//                        last chunk, subtract the scaled sums from A22.
// prev.a: the images of the previous panel, whose update of these tiles was
// deferred: its chunks run first and its sums are rescaled (exactly) to this
// panel's scales. Every wait is bounded; a role that times out raises the
// status and flags the others, and each waits (bounded) for its own copies and
// MMAs before the CTA frees its tensor memory.
__global__ void __launch_bounds__(OZ_THREADS, 1)
    oz_update_kernel(Batch b, int k0, OzSet cur, OzSet prev, OzStride st, int nsys, int* status, int ti0, int nti,
                     int tj0, int ntc) {
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OZ_SLOTS * OZ_SLOT);
  // full[8], empty[8], acc_full[4], acc_empty[4], drain; then the TMEM address
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * OZ_SLOTS + 2 * OZ_ACC + 1);
  __shared__ volatile int s_err;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[OZ_SLOTS]);
  const uint32_t accf0 = smem_u32(&bars[2 * OZ_SLOTS]), acce0 = smem_u32(&bars[2 * OZ_SLOTS + OZ_ACC]);
  const uint32_t drain = smem_u32(&bars[2 * OZ_SLOTS + 2 * OZ_ACC]);
  const int r1 = k0 + LU_OUTER;
  const long long total = (long long)nti * ntc * nsys;
  const int nch = prev.a ? 2 * OZ_NCH : OZ_NCH;
  auto tile = [&](long long t, int& z, int& trow, int& tcol) {
    z = (int)(t / ((long long)nti * ntc));
    const int rem = (int)(t % ((long long)nti * ntc));
    trow = ti0 + rem / ntc;
    tcol = tj0 + rem % ntc;
    const int rest = b.order(z) - r1;
    return rest > 0 && trow * OZ_M < rest && tcol * OZ_N < rest;
  };
  if (threadIdx.x == 0) {
    s_err = 0;
    for (int i = 0; i < 2 * OZ_SLOTS; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * i));
    for (int i = 0; i < OZ_ACC; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(accf0 + 8 * i));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(acce0 + 8 * i), "r"(OZ_EPI));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(drain));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(OZ_ACC * 2 * OZ_N));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  auto fail = [&] {
    atomicCAS(status, 0, ST_TC_TIMEOUT);
    s_err = 1;
  };
  // The slot of the p-th loaded slice of a chunk, the same sequence in the
  // producer and the issuer: first the spare slot, then the slots of the
  // previous chunk's slices 6, 5, .. 1 as their diagonals end; the slot of
  // slice 0 becomes the spare. `map` holds slice i's slot in nibble i, the
  // spare in nibble 7.
  auto next_map = [](uint32_t map) {
    uint32_t m = 0;
#pragma unroll
    for (int p = 0; p < OZ_S; ++p) {
      const uint32_t slot = (map >> (4 * (7 - p))) & 0xf;   // nibble 7 (spare), then 6 .. 1
      m |= slot << (4 * ((OZ_ORDER >> (4 * p)) & 0xf));
    }
    return m | ((map & 0xf) << 28);
  };
  constexpr uint32_t MAP0 = 0x76543210u;

  if (warp == 0 && lane == 0) {
    // producer
    const uint32_t s0 = smem_u32(smem);
    uint32_t map = MAP0, used = 0, eph = 0, fph = 0;   // slots loaded so far; parities of the next empty / last full wait
    bool ok = true;
    for (long long t = blockIdx.x; t < total && ok && !s_err; t += gridDim.x) {
      int z, trow, tcol;
      if (!tile(t, z, trow, tcol)) continue;
      for (int c = 0; c < nch && ok; ++c) {
        // the previous panel's trailing block starts 128 rows and columns earlier
        const bool pv = prev.a && c < OZ_NCH;
        const OzSet& s = pv ? prev : cur;
        const unsigned char* ga = s.a + z * st.a + ((long long)(trow + (pv ? 1 : 0)) * OZ_NCH + c % OZ_NCH) * OZ_S * OZ_A;
        const unsigned char* gb =
            s.b + z * st.b + ((long long)(tcol + (pv ? OZ_M / OZ_N : 0)) * OZ_NCH + c % OZ_NCH) * OZ_S * OZ_B;
        map = next_map(map);
        for (int p = 0; p < OZ_S; ++p) {
          const int i = (OZ_ORDER >> (4 * p)) & 0xf, q = (map >> (4 * i)) & 0xf;
          if ((used >> q) & 1) {
            if (!(ok = mbar_wait_suspend(empty0 + 8 * q, (eph >> q) & 1))) break;
            eph ^= 1u << q;
            fph ^= 1u << q;
          }
          used |= 1u << q;
          const uint32_t dst = s0 + q * OZ_SLOT, bar = full0 + 8 * q;
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(OZ_SLOT) : "memory");
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           dst),
                       "l"(ga + i * OZ_A), "r"(OZ_A), "r"(bar)
                       : "memory");
          asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           dst + OZ_A),
                       "l"(gb + i * OZ_B), "r"(OZ_B), "r"(bar)
                       : "memory");
        }
      }
    }
    if (!ok) fail();
    // copies in flight land before the CTA can leave: the last load of each slot
    for (int q = 0; q < OZ_SLOTS; ++q)
      if ((used >> q) & 1) mbar_wait_suspend(full0 + 8 * q, (fph >> q) & 1);
  } else if (warp == 1 && lane == 0) {
    // MMA issuer
    const uint32_t s0 = smem_u32(smem);
    const uint64_t da0 = umma_desc(s0, 128, OZ_ASBO), db0 = umma_desc(s0 + OZ_A, 128, OZ_BSBO);
    uint32_t map = MAP0, fph = 0;   // parity of the next full wait per slot
    long long g = 0;                // diagonals issued
    bool ok = true;
    for (long long t = blockIdx.x; t < total && ok && !s_err; t += gridDim.x) {
      int z, trow, tcol;
      if (!tile(t, z, trow, tcol)) continue;
      for (int c = 0; c < nch && ok; ++c) {
        map = next_map(map);
        uint32_t have = 0;   // slices of this chunk known to have landed
        for (int s = OZ_D - 1; s >= 0 && ok; --s, ++g) {
          const int buf = (int)(g % OZ_ACC);
          if (g >= OZ_ACC && !(ok = mbar_wait_suspend(acce0 + 8 * buf, (uint32_t)((g / OZ_ACC - 1) & 1)))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t tm = tmem + (uint32_t)(buf * 2 * OZ_N);
          const int lo = max(0, s - (OZ_S - 1)), cnt = s - 2 * lo + 1;   // pairs (lo, s - lo) .. (s - lo, lo)
          for (int m = 0; m < cnt; ++m) {
            // from the middle outwards on the first diagonal (the order the slices arrive in)
            const int mid = cnt / 2, i = lo + (s == OZ_D - 1 ? ((m & 1) ? mid + m / 2 : mid - 1 - m / 2) : m), j = s - i;
            const int qa = (map >> (4 * i)) & 0xf, qb = (map >> (4 * j)) & 0xf;
            for (int h = 0; h < 2 && ok; ++h) {
              const int sl = h ? j : i, q = h ? qb : qa;
              if (!((have >> sl) & 1)) {
                if (!(ok = mbar_wait_suspend(full0 + 8 * q, (fph >> q) & 1))) break;
                fph ^= 1u << q;
                have |= 1u << sl;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              }
            }
            if (!ok) break;
            const uint64_t da = da0 + (uint64_t)((qa * OZ_SLOT) >> 4), db = db0 + (uint64_t)((qb * OZ_SLOT) >> 4);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)   // Ar against (Br, Bi), then Ai against (-Bi, Br)
              oz_mma(tm, da + (uint64_t)((kk * 256) >> 4), db + (uint64_t)(((kk < 2 ? OZ_PLANE : 0) + (kk & 1) * 256) >> 4),
                     (m > 0 || kk > 0) ? 1u : 0u);
          }
          if (!ok) break;
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(accf0 +
                                                                                                           8 * buf)
                       : "memory");
          if (s < OZ_S)   // slice s is in no diagonal below
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             empty0 + 8 * ((map >> (4 * s)) & 0xf))
                         : "memory");
        }
      }
    }
    if (!ok) fail();
    // every MMA issued has completed before the tensor memory is freed
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(drain) : "memory");
    mbar_wait_suspend(drain, 0);
  } else if (warp >= 2) {
    // epilogue: thread = TMEM lane (row), 32 complex columns of the tile
    const int lq = warp & 3, half = (warp - 2) >> 2;
    const int row = lq * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)(32 * half);
    long long g = 0;
    bool ok = true;
    for (long long t = blockIdx.x; t < total && ok; t += gridDim.x) {
      if (__shfl_sync(0xffffffffu, s_err, 0)) break;
      int z, trow, tcol;
      if (!tile(t, z, trow, tcol)) continue;
      const int n = b.order(z);
      const int gr = r1 + trow * OZ_M + row, c0 = r1 + tcol * OZ_N + 32 * half;
      const int ncol = min(32, n - c0);
      double2* C = b.sys(z) + gr + (long long)n * c0;
      // the tile comes into L2 while its products run
      if (gr < n && (lane & 7) == 0)
        for (int j = 0; j < ncol; ++j) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + (long long)n * j));
      double ar[32], ai[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) ar[j] = ai[j] = 0.;
      for (int c = 0; c < nch && ok; ++c) {
        if (prev.a && c == OZ_NCH) {   // the deferred panel's sums in this panel's scales
          const double* pr = prev.ra + z * st.s + (trow + 1) * OZ_M + row;
          const double* pc = prev.cb + z * st.s + tcol * OZ_N + OZ_M + 32 * half;
          const double* cc = cur.cb + z * st.s + tcol * OZ_N + 32 * half;
          const double rr = *pr / cur.ra[z * st.s + trow * OZ_M + row];
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const double f = rr * (pc[j] / cc[j]);
            ar[j] *= f;
            ai[j] *= f;
          }
        }
        double wt = 1.;   // weight of the diagonal: 256^(7 - s)
        for (int s = OZ_D - 1; s >= 0; --s, ++g, wt *= 256.) {
          const int buf = (int)(g % OZ_ACC);
          const bool got = mbar_wait_suspend(accf0 + 8 * buf, (uint32_t)((g / OZ_ACC) & 1));
          if (!(ok = __all_sync(0xffffffffu, got))) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t ta = tl + (uint32_t)(buf * 2 * OZ_N);
          uint32_t v[16];
          // INT32 -> FP64 by its bits: 2^52 + 2^31 + v, exactly
          auto value = [](uint32_t x) { return __hiloint2double(0x43300000, (int)(x ^ 0x80000000u)) - 4503601774854144.; };
#pragma unroll
          for (int h = 0; h < 4; ++h) {   // Re columns 0..15, 16..31, Im columns 0..15, 16..31
            tmem_ld16(ta + (h >> 1) * OZ_N + (h & 1) * 16, v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (h == 3) {   // the accumulator is read: release it
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acce0 + 8 * buf) : "memory");
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              double& a = h < 2 ? ar[16 * (h & 1) + j] : ai[16 * (h & 1) + j];
              a = fma(value(v[j]), wt, a);
            }
          }
        }
      }
      if (!ok) break;
      if (gr < n) {
        const double rs = cur.ra[z * st.s + trow * OZ_M + row];
        const double* cc = cur.cb + z * st.s + tcol * OZ_N + 32 * half;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          double2 v[4];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (4 * q + j < ncol) v[j] = C[(long long)n * (4 * q + j)];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (4 * q + j < ncol) {
              const double f = -rs * cc[4 * q + j];
              v[j].x = fma(ar[4 * q + j], f, v[j].x);
              v[j].y = fma(ai[4 * q + j], f, v[j].y);
              C[(long long)n * (4 * q + j)] = v[j];
            }
        }
      }
    }
    if (!ok) fail();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(OZ_ACC * 2 * OZ_N));
}

// images of the panel [k0, k0 + 128) into s
inline void oz_prep(const OzSet& s, const OzStride& st, Batch b, int k0, int nsys, cudaStream_t stream,
                    long long& launches) {
  const int rest = b.n - k0 - LU_OUTER;
  if (rest <= 0) return;
  const int per = (rest + OZ_M - 1) / OZ_M * (OZ_M / 32);
  oz_prep_kernel<<<dim3(2 * per, 1, nsys), OZP_THREADS, 0, stream>>>(b, k0, s, st, per);
  ++launches;
}

// A[r1 + 128 i0 :, r1 + 128 j0 :] of the panel's trailing block, `ni` x `nj`
// blocks of 128 (negative: to the end), from the images in cur (and the
// deferred panel's in prev)
inline void oz_apply(const OzSet& cur, const OzSet& prev, const OzStride& st, Batch b, int k0, int nsys,
                     cudaStream_t stream, long long& launches, int* status, TcTiles tl) {
  const int rest = b.n - k0 - LU_OUTER;
  if (rest <= 0) return;
  const int nt = (rest + OZ_M - 1) / OZ_M, nc = (rest + OZ_N - 1) / OZ_N;
  constexpr int CPB = OZ_M / OZ_N;   // column tiles per block of 128
  const int nti = std::min(tl.nti < 0 ? nt - tl.ti0 : tl.nti, nt - tl.ti0);
  const int tj0 = CPB * tl.tj0;
  const int ntc = std::min(tl.ntc < 0 ? nc - tj0 : CPB * tl.ntc, nc - tj0);
  if (nti <= 0 || ntc <= 0) return;
  static std::atomic<unsigned long long> attr{0};
  static int sms = 0;
  once_per_device(attr, [] {
    cudaFuncSetAttribute(oz_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM);
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  });
  const long long tiles = (long long)nti * ntc * nsys;
  const int grid = (int)std::min<long long>(tiles, sms > 0 ? sms : 148);
  oz_update_kernel<<<grid, OZ_THREADS, OZ_SMEM, stream>>>(b, k0, cur, prev, st, nsys, status, tl.ti0, nti, tj0, ntc);
  ++launches;
}

}  // namespace nb200
