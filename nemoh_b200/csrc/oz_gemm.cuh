// Trailing update of the FP64 LU on the tensor cores (tcgen05, sm_100a).
//
//     A22 <- A22 - L21 * U12        (complex FP64, inner dimension K = 128 per panel)
//
// B200's FP64 pipe multiplies at 30 TFLOP/s (measured); its INT8 tensor pipe is
// two orders of magnitude wider and exact. So each operand is split into
// integer slices (the error-free splitting of Ozaki, Ogita, Oishi and Rump):
// row r of L21 (column c of U12) gets one power-of-two scale 2^e above its
// largest component over the panel, every component becomes the integer
// V = rint(x 2^(62 - e)), |V| <= 2^62, and V its eight balanced base-256 digits
//     V = sum_t d_t 256^t,  d_t in [-128, 127].
// Slice i holds the digits of weight 256^(7 - i). Products of equal i + j share
// an INT32 accumulator (a diagonal) over K = 128 complex, exactly (at most 8
// products of 256 terms of 2^14: 2^25), and the diagonals are summed in FP64 with
// their powers of 256.
//
// Diagonals i + j <= 7 are kept (36 slice products; slice 7 only meets slice 0).
// A component down to 2^-9 of its row's largest is held with all its 53 bits,
// the rounding of a smaller one is 2^-63 of the scale at most; what is dropped is
// below 2^-58 of the product of the two scales per k. Both are relative to a row's
// and a column's largest components, not to the entry that they update, which is
// far smaller where the panel's columns couple weakly with one another. Measured
// against 80-bit arithmetic, FP64 multiply-add chain / this form / seven slices
// of 55 bits (34 products), the 90% and 99.9% quantiles of the factors' errors
// relative to each entry: cylinder of 528 panels at 1 rad/s 8.8e-16, 2.9e-15 /
// 7.1e-16, 1.8e-15 / 7.1e-16, 1.9e-15, at 2.5 rad/s 8.6e-16, 8.6e-15 / 7.8e-16,
// 4.1e-15 / 8.3e-16, 1.4e-14; box of 100 x 20 x 10 m and 608 panels at 2.5 rad/s (90%)
// 1.4e-15 / 1.3e-15 / 7.1e-15 and its sources (99%) 3.4e-15 / 3.1e-15 / 4.3e-15.
// The errors relative to the largest entries agree within 6% in all three.
//
// How weakly the columns of a panel may couple is bounded by oz_wide: in a mesh
// whose numbering mixes a small hull with a large one far away the entries that
// couple them lose digits (1:20 hulls of 334 panels, 200 m apart, taking turns:
// sources' 99% quantile 2.0e-13 / 6.6e-13 / 7.8e-12; 1:100 and 20 m apart 9.2e-14 /
// 2.3e-12 / 3.5e-11). Such panels are updated on the FP64 pipe.
//
// The complex product is real: A as [Ar | Ai] along k, B as the planes
// [-Bi; Br; Bi] of 64 columns each, of which Ar multiplies (Br, Bi) and Ai
// multiplies (-Bi, Br): two neighbouring planes each, so B needs three planes
// instead of four.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "linalg.cuh"
#include "tc_gemm.cuh"

namespace nb200 {

constexpr int OZ_S = 8;                          // slices per operand
constexpr int OZ_BITS = 62;                      // |V| <= 2^62
constexpr int OZ_M = 128;                        // rows per tile
constexpr int OZ_N = 64;                         // complex columns per tile (128 accumulator columns: Re, Im)
constexpr int OZ_KC = 64;                        // complex k per chunk
constexpr int OZ_NCH = LU_OUTER / OZ_KC;         // chunks per panel
constexpr int OZ_A = OZ_M * 2 * OZ_KC;           // 16 KB: one slice of an A chunk
constexpr int OZ_PLANE = OZ_N * OZ_KC;           // 4 KB: one plane of a B slice
constexpr int OZ_B = 3 * OZ_PLANE;               // 12 KB: one slice of a B chunk
constexpr int OZ_ASBO = 2 * OZ_KC * 8;           // bytes between 8-row groups of an A slice
constexpr int OZ_BSBO = OZ_KC * 8;               // and of a B plane
constexpr int OZ_SLOT = OZ_A + OZ_B;             // 28 KB: one slice of both operands
constexpr int OZ_SLOTS = 8;
constexpr int OZ_ACC = 4;                        // accumulators of 128 tensor-memory columns
constexpr int OZ_EPI_WARPS = 16;
constexpr int OZ_THREADS = 128 + 32 * OZ_EPI_WARPS;   // producer, two MMA issuers, an idle warp; the epilogue's
constexpr int OZ_EC = OZ_N / (OZ_EPI_WARPS / 4);   // complex columns per epilogue thread
constexpr int OZ_BATCH = 2;                        // of them loaded at once
constexpr int OZ_SMEM = OZ_SLOTS * OZ_SLOT + 256 + 2 * 2 * OZ_N * (int)sizeof(double);
// Smallest scale exponent: components of rows and columns whose largest is below
// 2^-250 lose digits below 2^-313. The factors of influence matrices, whose
// diagonals are O(1), have no such rows but zero ones.
constexpr int OZ_EMIN = -250;
// Trailing entries of a batch (summed over its systems that the panel has not
// finished) from which an update takes this path; below it the FP64 pipe's one
// launch is as fast as the images and the update, which then cover few SMs. LU in
// ms, FP64 pipe / this path: 10 systems of 420 panels (0.9 M entries) 0.59 / 0.61, 4
// of 588 (0.8 M) 0.79 / 0.86, 2 of 894 (1.2 M) 1.00 / 1.04, 20 of 420 (1.7 M) 0.69 /
// 0.66, 4 of 894 (2.3 M) 1.25 / 1.16, 2 of 1,430 (3.4 M) 2.09 / 1.86, 20 of 588
// (4.2 M) 1.19 / 1.00, 1 of 2,380 (5.1 M) 4.05 / 3.21, 20 of 2,380 (101 M) 37.0 / 16.8.
// Ragged: 1 of 1,400 with 19 of 200 (1.7 M after the first panel) 1.77 / 1.75, 2 of 1,100
// with 20 of 200 (2.0 M) 1.50 / 1.46, 1 of 1,800 with 20 of 200 (2.9 M) 2.62 / 2.37, 3 of 1,000
// with 6 of 500 (3.1 M) 1.49 / 1.36, 1 of 3,000 with 40 of 200 (8.5 M) 6.54 / 4.76, 4 of 2,600 with 8
// of 1,200 and 12 of 400 (35 M) 13.6 / 7.6.
constexpr double OZ_MIN_ENTRIES = 1.5e6;
// Tiles of a full update (summed likewise) from which panel pairs are merged (four
// per SM): the merged form reads and writes the trailing block once per pair, the
// corner update it needs is a launch of one tile's latency more. LU in ms, never
// merged / from 600 tiles / from 148: 20 systems of 420 0.66 / 0.66 / 0.66, 10 of 894
// 1.46 / 1.44 / 1.41, 1 of 2,380 3.25 / 3.21 / 3.20, 20 of 2,380 18.1 / 16.8 / 16.8.
constexpr long long OZ_MERGE_TILES = 600;

// Panels of the LU (128 consecutive panels of the mesh) whose update stays on the
// FP64 pipe: those in which the square of the bounding box's diagonal is more than
// OZ_MAX_SPREAD times the smallest area. A panel of area a couples with one at a
// distance d by a / (2 pi d^2) at the most, its neighbours with it by 0.1 or so; the
// digits are relative to the latter. Contiguous parts of one hull stay below:
// barges, cylinders and spheres of 300 to 4,000 panels and fleets of random hulls
// of up to 3,000 reach 3.5e4, typically 3e2 to 3e3. Hulls that take turns in the
// numbering (90% and 99.9% quantiles of the factors' errors per entry at 2.5 rad/s,
// FP64 chain / slices): equal ones 100 m apart, 4e4: 1.1e-15, 1.6e-14 / 1.1e-15,
// 2.5e-14; 300 m, 4e5: 1.4e-15, 1.9e-14 / 1.9e-15, 4.1e-13.
constexpr double OZ_MAX_SPREAD = 4e4;
inline std::vector<char> oz_wide(int nfa, const double* xyz, const int* m1234) {
  std::vector<char> wide((nfa + LU_OUTER - 1) / LU_OUTER);
  for (size_t b = 0; b < wide.size(); ++b) {
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300}, area2 = 1e300, d2 = 0.;
    for (int i = (int)b * LU_OUTER; i < std::min(nfa, ((int)b + 1) * LU_OUTER); ++i) {
      const double* v[4];
      for (int k = 0; k < 4; ++k) {
        v[k] = xyz + 3 * (size_t)(m1234[4 * i + k] - 1);
        for (int c = 0; c < 3; ++c) {
          lo[c] = std::min(lo[c], v[k][c]);
          hi[c] = std::max(hi[c], v[k][c]);
        }
      }
      double p[3], q[3], a2 = 0.;   // the diagonals, the square of twice the area
      for (int c = 0; c < 3; ++c) p[c] = v[2][c] - v[0][c], q[c] = v[3][c] - v[1][c];
      for (int c = 0; c < 3; ++c) {
        const double x = p[(c + 1) % 3] * q[(c + 2) % 3] - p[(c + 2) % 3] * q[(c + 1) % 3];
        a2 += x * x;
      }
      area2 = std::min(area2, a2);
    }
    for (int c = 0; c < 3; ++c) d2 += (hi[c] - lo[c]) * (hi[c] - lo[c]);
    wide[b] = !(d2 <= OZ_MAX_SPREAD * 0.5 * std::sqrt(area2));
  }
  return wide;
}

// The schedule of a tile. Its 72 slice products run in four phases: diagonals 7 ..
// 4 of both chunks into the four accumulators, then diagonals 0 .. 3 of both
// chunks (slices 0 .. 3, loaded again), so that an accumulator is drained once per
// phase pair and not once per chunk: the FP64 pipe and the tensor pipe do not run
// at the same time (measured: 384 k cycles of DFMA and 410 k of MMA take 833 k
// together), and every drained value costs FP64 work. Slice 7 of a chunk, which
// only meets slice 0, borrows a slot that is free or retires at once.
// Each step is one slice product (A slice i, B slice j) of a phase. The order lets
// slices retire early and lets the accumulators finish in pairs, (0, 1) before
// (2, 3), which are drained and free again before the next phase pair meets them;
// slices of one phase lie in other slots than those of the next where the same
// slot would free up too late. A load is (slice, slot).
struct OzStep {
  signed char i, j;      // slices of A and B
  signed char slot_i, slot_j;
  signed char acc;       // accumulator
  signed char first;     // first product of its accumulator
  short need;            // slots to wait for, as a bit mask
  short retire;          // slots no later step of the phase reads, as a bit mask
  signed char full;      // accumulators finished, as a bit mask
};
template <int N>
struct OzPhase {
  OzStep s[N];
  int count;   // steps in use
};
// The steps of one issuer (accumulators `mine`, a bit mask) of a phase.
// slots[i]: slot of slice i (nsl slices); pairs: (i, j) in order; low: diagonals 0
// .. 3 (accumulator i + j), else 7 .. 4 (accumulator 7 - i - j); begin / end: the
// first / last chunk of the phase pair. Both issuers wait for and release every
// slot of the phase (a slot's barrier counts two releases), one that this issuer
// does not read with its first step after the other's last read, or with its last.
template <int N>
constexpr OzPhase<N> oz_phase(const int (&pairs)[N][2], const int (&slots)[OZ_S], int nsl, bool low, bool begin,
                              bool end, int mine) {
  OzPhase<N> p{};
  int all = 0;
  for (int i = 0; i < nsl; ++i) all |= 1 << slots[i];
  int seen = 0, used = 0, reads = 0;
  for (int k = 0; k < N; ++k)
    if ((mine >> (low ? pairs[k][0] + pairs[k][1] : 7 - pairs[k][0] - pairs[k][1])) & 1)
      reads |= (1 << slots[pairs[k][0]]) | (1 << slots[pairs[k][1]]);
  for (int k = 0; k < N; ++k) {
    const int i = pairs[k][0], j = pairs[k][1], acc = low ? i + j : 7 - i - j;
    if (!((mine >> acc) & 1)) continue;
    OzStep& t = p.s[p.count++];
    t.i = (signed char)i;
    t.j = (signed char)j;
    t.slot_i = (signed char)slots[i];
    t.slot_j = (signed char)slots[j];
    t.acc = (signed char)acc;
    t.first = begin && !((used >> acc) & 1);
    used |= 1 << acc;
    int m = (1 << slots[i]) | (1 << slots[j]);
    int later = 0, open = 0;
    for (int q = k + 1; q < N; ++q) {
      const int a = low ? pairs[q][0] + pairs[q][1] : 7 - pairs[q][0] - pairs[q][1];
      if (!((mine >> a) & 1)) continue;
      later |= (1 << slots[pairs[q][0]]) | (1 << slots[pairs[q][1]]);
      open |= 1 << a;
    }
    int ahead = 0;   // slots that either issuer reads from here on
    for (int q = k; q < N; ++q) ahead |= (1 << slots[pairs[q][0]]) | (1 << slots[pairs[q][1]]);
    m |= (later == 0 ? all : all & ~(reads | ahead)) & ~seen;
    t.need = (short)(m & ~seen);
    seen |= m;
    t.retire = (short)(m & ~later);
    t.full = (signed char)(end && !((open >> acc) & 1) ? 1 << acc : 0);
  }
  return p;
}
constexpr int OZ_P0[26][2] = {{1, 6}, {6, 1}, {1, 5}, {5, 1}, {1, 4}, {4, 1}, {0, 7}, {7, 0}, {0, 6},
                              {6, 0}, {0, 5}, {5, 0}, {0, 4}, {4, 0}, {2, 5}, {5, 2}, {2, 4}, {4, 2},
                              {2, 2}, {3, 4}, {4, 3}, {3, 3}, {2, 3}, {3, 2}, {1, 3}, {3, 1}};
constexpr int OZ_P1[26][2] = {{1, 6}, {6, 1}, {1, 5}, {5, 1}, {0, 6}, {6, 0}, {2, 5}, {5, 2}, {2, 4},
                              {4, 2}, {0, 7}, {7, 0}, {3, 4}, {4, 3}, {3, 3}, {0, 5}, {5, 0}, {1, 4},
                              {4, 1}, {2, 3}, {3, 2}, {0, 4}, {4, 0}, {1, 3}, {3, 1}, {2, 2}};
constexpr int OZ_P2[10][2] = {{0, 0}, {0, 1}, {1, 0}, {1, 1}, {0, 2}, {2, 0}, {1, 2}, {2, 1}, {0, 3}, {3, 0}};
constexpr int OZ_P3[10][2] = {{0, 0}, {0, 1}, {1, 0}, {0, 2}, {2, 0}, {1, 1}, {1, 2}, {2, 1}, {0, 3}, {3, 0}};
constexpr int OZ_L0[OZ_S] = {0, 1, 2, 3, 4, 5, 6, 7}, OZ_L1[OZ_S] = {0, 7, 2, 3, 4, 5, 6, 1},
              OZ_L2[OZ_S] = {6, 1, 5, 4}, OZ_L3[OZ_S] = {0, 7, 2, 3};
// Two warps issue, each with two of the accumulators: an MMA is handed over only
// about when the one before it starts (measured: a pause of 200 cycles after every
// four MMAs costs 219), so one issuer's waits and releases would leave the tensor
// pipe idle; the other's MMAs fill them.
constexpr int OZ_WHO0 = (1 << 0) | (1 << 3), OZ_WHO1 = (1 << 1) | (1 << 2);
template <int WHO>
struct OzPlan {
  static constexpr OzPhase<26> p0 = oz_phase(OZ_P0, OZ_L0, 8, false, true, false, WHO);
  static constexpr OzPhase<26> p1 = oz_phase(OZ_P1, OZ_L1, 8, false, false, true, WHO);
  static constexpr OzPhase<10> p2 = oz_phase(OZ_P2, OZ_L2, 4, true, true, false, WHO);
  static constexpr OzPhase<10> p3 = oz_phase(OZ_P3, OZ_L3, 4, true, false, true, WHO);
};
// the loads of a tile in the order their slots free up
constexpr int OZ_LOADS = 24;
constexpr signed char OZ_LOAD[OZ_LOADS][3] = {   // slice, slot, chunk
    {1, 1, 0}, {6, 6, 0}, {5, 5, 0}, {4, 4, 0}, {7, 7, 0}, {0, 0, 0}, {2, 2, 0}, {3, 3, 0},
    {1, 7, 1}, {6, 6, 1}, {0, 0, 1}, {5, 5, 1}, {4, 4, 1}, {2, 2, 1}, {7, 1, 1}, {3, 3, 1},
    {0, 6, 0}, {1, 1, 0}, {2, 5, 0}, {3, 4, 0},
    {0, 0, 1}, {1, 7, 1}, {2, 2, 1}, {3, 3, 1}};

// Operand images and scales of two panels (the update of one panel may be
// merged into the next one's): per set and system ceil(n / 128) row tiles and 2
// ceil(n / 128) column tiles of OZ_NCH chunks of OZ_S slices; scales one per row,
// then one per column.
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
  bool grows(int ns, int n) const {
    const size_t t = 2 * (size_t)ns * ((n + OZ_M - 1) / OZ_M);
    return t * OZ_NCH * OZ_S * OZ_A > have_a || t * 2 * OZ_NCH * OZ_S * OZ_B > have_b ||
           t * 2 * OZ_M * sizeof(double) > have_sc;
  }
  // all of the images or none of them
  cudaError_t ensure(int ns, int n, bool headroom = false) {
    tiles = (n + OZ_M - 1) / OZ_M;
    nsys = ns;
    const size_t t = 2 * (size_t)ns * tiles;
    cudaError_t e = grow_alloc(reinterpret_cast<void**>(&a), &have_a, t * OZ_NCH * OZ_S * OZ_A, headroom);
    if (!e) e = grow_alloc(reinterpret_cast<void**>(&b), &have_b, t * 2 * OZ_NCH * OZ_S * OZ_B, headroom);
    if (!e) e = grow_alloc(reinterpret_cast<void**>(&sc), &have_sc, t * 2 * OZ_M * sizeof(double), headroom);
    if (e) release();
    return e;
  }
};
inline size_t oz_bytes_per_system(size_t n) {
  const size_t t = 2 * ((n + OZ_M - 1) / OZ_M);
  return t * (OZ_NCH * OZ_S * (size_t)(OZ_A + 2 * OZ_B) + 2 * OZ_M * sizeof(double));
}

// The images as the kernels take them (bases of the launch's first system):
// strides are per system.
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

// 16 components scaled by 2^(62 - e): their digits, slice by slice, as 16-byte
// rows out(i, uint4). V + 0x8080..80 has the digits offset by 128 as its bytes,
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
          ((unsigned long long)v + 0x8080808080808080ull) ^ 0x8080808080808080ull;
      lo[j] = (uint32_t)u;
      hi[j] = (uint32_t)(u >> 32);
    }
    // byte t of the four values, in order, is the word of slice 7 - t
    auto quad = [](const uint32_t* v, uint32_t& b0, uint32_t& b1, uint32_t& b2, uint32_t& b3) {
      const uint32_t p = __byte_perm(v[0], v[1], 0x5140), q2 = __byte_perm(v[2], v[3], 0x5140);
      const uint32_t r = __byte_perm(v[0], v[1], 0x7362), s = __byte_perm(v[2], v[3], 0x7362);
      b0 = __byte_perm(p, q2, 0x5410);
      b1 = __byte_perm(p, q2, 0x7632);
      b2 = __byte_perm(r, s, 0x5410);
      b3 = __byte_perm(r, s, 0x7632);
    };
    quad(lo, w[7][q], w[6][q], w[5][q], w[4][q]);
    quad(hi, w[3][q], w[2][q], w[1][q], w[0][q]);
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
// 256^7 .. 1 in units of 256^7, 2^28 of each operand. A row with a
// NaN or an infinity makes every result of the row NaN.
__device__ __forceinline__ double oz_scale(unsigned mag, int e) {
  return mag >= 0x7ff00000u ? __longlong_as_double(0x7ff8000000000000ll) : oz_pow2(e - 34);
}

// Images of the panel [k0, k0 + 128): L21 = A[r1:n, k0:r1] and U12 = A[k0:r1,
// r1:n], r1 = k0 + 128. Blocks [0, na): 32 rows of L21, thread = (row, 16 k);
// the others: 32 columns of U12, thread = (column, 16 k). Reads 16 B and writes
// 16 B (L21) or 24 B (U12) per entry (two systems of 2,252 rows: 14.5 us), bound by HBM and the FP64 -> INT64
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
  const double sc = oz_pow2(OZ_BITS - e);
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

__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(addr));
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t* a, uint32_t* b) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i) asm volatile("" : "+r"(a[i]), "+r"(b[i]));   // the values are there only now
}

// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
  uint32_t e;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(e));
  return e != 0;
}

// Step K of a phase: waits for the slices and the accumulator it meets first,
// issues its four MMAs, and releases the slots and accumulators it is the last of.
// sync.full(slot) / sync.empty(acc) wait, uniformly over the warp.
template <const auto& PH, int K, class Sync>
__device__ __forceinline__ bool oz_step(uint32_t tmem, uint64_t da, uint64_t db, bool issue, uint32_t empty0,
                                        uint32_t accf0, Sync& sync) {
  constexpr OzStep t = PH.s[K];
  if (t.first && !sync.empty(t.acc)) return false;
#pragma unroll
  for (int q = 0; q < OZ_SLOTS; ++q)
    if ((t.need >> q) & 1)
      if (!sync.full(q)) return false;
  if (issue) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)   // Ar against (Br, Bi), then Ai against (-Bi, Br)
      oz_mma(tmem + t.acc * 2 * OZ_N, da + (uint64_t)((t.slot_i * OZ_SLOT + kk * 256) >> 4),
             db + (uint64_t)((t.slot_j * OZ_SLOT + (kk < 2 ? OZ_PLANE : 0) + (kk & 1) * 256) >> 4),
             (kk > 0 || !t.first) ? 1u : 0u);
    if (t.full)
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(accf0 +
                                                                                                       8 * t.acc)
                   : "memory");
#pragma unroll
    for (int q = 0; q < OZ_SLOTS; ++q)
      if ((t.retire >> q) & 1)
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(empty0 + 8 * q)
                     : "memory");
  }
  __syncwarp();
  return true;
}
template <const auto& PH, class Sync, int... K>
__device__ __forceinline__ bool oz_steps(std::integer_sequence<int, K...>, uint32_t tmem, uint64_t da, uint64_t db,
                                         bool issue, uint32_t empty0, uint32_t accf0, Sync& sync) {
  return (oz_step<PH, K>(tmem, da, db, issue, empty0, accf0, sync) && ...);
}
template <const auto& PH, class Sync>
__device__ __forceinline__ bool oz_run(uint32_t tmem, uint64_t da, uint64_t db, bool issue, uint32_t empty0,
                                       uint32_t accf0, Sync& sync) {
  return oz_steps<PH>(std::make_integer_sequence<int, PH.count>{}, tmem, da, db, issue, empty0, accf0, sync);
}

// The waits of the MMA issuer (by every lane of its warp).
struct OzSync {
  uint32_t full0, acce0;
  uint32_t fph = 0;    // parity of the next full wait per slot
  uint32_t aph = 0;    // parity of the next empty wait per accumulator
  uint32_t used = 0;   // accumulators used before
  __device__ __forceinline__ bool full(int q) {
    const bool got = mbar_wait_suspend(full0 + 8 * q, (fph >> q) & 1);
    fph ^= 1u << q;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return __all_sync(0xffffffffu, got) != 0;
  }
  __device__ __forceinline__ bool empty(int a) {
    bool got = true;
    if ((used >> a) & 1) {
      got = mbar_wait_suspend(acce0 + 8 * a, (aph >> a) & 1);
      aph ^= 1u << a;
    }
    used |= 1u << a;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    return __all_sync(0xffffffffu, got) != 0;
  }
};

// Load L of a tile's schedule: waits until its slot is free and copies a slice of
// A and B into it. used: slots loaded before; eph, fph: parity of the next empty
// wait and of the last load per slot.
template <int L>
__device__ __forceinline__ bool oz_load(const unsigned char* ga, const unsigned char* gb, uint32_t s0, uint32_t full0,
                                        uint32_t empty0, uint32_t& used, uint32_t& eph, uint32_t& fph) {
  constexpr int i = OZ_LOAD[L][0], q = OZ_LOAD[L][1], c = OZ_LOAD[L][2];
  if ((used >> q) & 1) {
    if (!mbar_wait_suspend(empty0 + 8 * q, (eph >> q) & 1)) return false;
    eph ^= 1u << q;
    fph ^= 1u << q;
  }
  used |= 1u << q;
  const uint32_t dst = s0 + q * OZ_SLOT, bar = full0 + 8 * q;
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(OZ_SLOT) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(ga + (c * OZ_S + i) * OZ_A), "r"(OZ_A), "r"(bar)
               : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst +
                                                                                                             OZ_A),
               "l"(gb + (c * OZ_S + i) * OZ_B), "r"(OZ_B), "r"(bar)
               : "memory");
  return true;
}
template <int... L>
__device__ __forceinline__ bool oz_load_tile(std::integer_sequence<int, L...>, const unsigned char* ga,
                                             const unsigned char* gb, uint32_t s0, uint32_t full0, uint32_t empty0,
                                             uint32_t& used, uint32_t& eph, uint32_t& fph) {
  return (oz_load<L>(ga, gb, s0, full0, empty0, used, eph, fph) && ...);
}

// a thread's row of the tile: C -= rs cc (ar + i ai), OZ_BATCH columns at a time
__device__ __forceinline__ void oz_subtract(double2* C, int n, int ncol, double rs, const double* cc, const double* ar,
                                            const double* ai) {
#pragma unroll
  for (int q = 0; q < OZ_EC; q += OZ_BATCH) {
    double2 v[OZ_BATCH];
    double2* p = C;
#pragma unroll
    for (int j = 0; j < OZ_BATCH; ++j, p += n)
      if (q + j < ncol) v[j] = *p;
#pragma unroll
    for (int j = 0; j < OZ_BATCH; ++j, C += n)
      if (q + j < ncol) {
        const double f = -rs * cc[q + j];
        v[j].x = fma(ar[q + j], f, v[j].x);
        v[j].y = fma(ai[q + j], f, v[j].y);
        *C = v[j];
      }
  }
}

// The update by tiles of 128 x 64 complex (nti row tiles, ntc column tiles) of
// every system, one persistent CTA per SM walking tile t, t + grid, ...:
//   warp 0 (one thread)  loads slices of A and B (28 KB) into the slots, in OZ_LOAD's order;
//   warps 1 and 2        issue the MMAs of their accumulators: the whole warp walks
//                        the phases, so that every address is warp-uniform, and one
//                        lane issues; the steps are written out (looked up step by
//                        step they took longer than their MMAs);
//   warps 4-19           add a finished pair of diagonals to the tile's FP64 sums
//                        (32 per thread, in registers; warp w the TMEM lanes 32 (w %
//                        4) .. and quarter (w - 4) / 4 of the columns) and, at the
//                        end, subtract the scaled sums from A22, while the next
//                        tile's first products run.
// prev.a: the images of the previous panel, whose update of these tiles was
// deferred: its products run first and its sums are rescaled (exactly) to this
// panel's scales. corner: the tiles of the next panel's columns and rows only.
// Every wait is bounded; a role that times out raises the status and flags the
// others, and each waits (bounded) for its own copies and MMAs before the CTA
// frees its tensor memory.
// What bounds it: the tensor pipe at 64 cycles an MMA (an N = 128 MMA reads its
// operands from shared memory at the port's 128 B a cycle), the FP64 and integer
// work of the drains, which takes tensor cycles, and the read-modify-write of A22,
// 256 KB per tile. Two systems of 2,252 trailing rows: 205 us per panel (1,296
// tiles, 18,400 cycles of MMAs each), 299 us for a merged pair, 27 us for a corner.
// With seven slices per operand (17,400 cycles) 198, 291 and 25 us, of which 113
// without drains and A22; a first form that drained every 64 complex k took 256 and
// 420 us, the FP64 pipe 830 us per panel.
__global__ void __launch_bounds__(OZ_THREADS, 1)
    oz_update_kernel(Batch b, int k0, OzSet cur, OzSet prev, OzStride st, int nsys, int* status, int nti, int ntc,
                     int corner) {
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OZ_SLOTS * OZ_SLOT);
  // full[8], empty[8], acc_full[4], acc_empty[4], drain; then the TMEM address
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * OZ_SLOTS + 2 * OZ_ACC + 1);
  // a tile's column scales and, in a merged update, the ratios of the deferred
  // panel's to them; two tiles' worth
  double(*s_col)[2][OZ_N] = reinterpret_cast<double(*)[2][OZ_N]>(smem + OZ_SLOTS * OZ_SLOT + 256);
  __shared__ volatile int s_err;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t full0 = smem_u32(&bars[0]), empty0 = smem_u32(&bars[OZ_SLOTS]);
  const uint32_t accf0 = smem_u32(&bars[2 * OZ_SLOTS]), acce0 = smem_u32(&bars[2 * OZ_SLOTS + OZ_ACC]);
  const uint32_t drain = smem_u32(&bars[2 * OZ_SLOTS + 2 * OZ_ACC]);
  const int r1 = k0 + LU_OUTER;
  // corner: only the first 128 columns (every row) and the first 128 rows
  constexpr int CW = LU_OUTER / OZ_N;   // column tiles of a panel's width
  const int per = corner ? CW * nti + max(0, ntc - CW) : nti * ntc;
  const long long total = (long long)per * nsys;
  const int parts = prev.a ? 2 : 1;
  auto tile = [&](long long t, int& z, int& trow, int& tcol) {
    z = (int)(t / per);
    const int rem = (int)(t % per);
    if (!corner) {
      trow = rem / ntc;
      tcol = rem % ntc;
    } else if (rem < CW * nti) {
      trow = rem / CW;
      tcol = rem % CW;
    } else {
      trow = 0;
      tcol = rem - CW * nti + CW;
    }
    const int rest = b.order(z) - r1;
    return rest > 0 && trow * OZ_M < rest && tcol * OZ_N < rest;
  };
  if (threadIdx.x == 0) {
    s_err = 0;
    for (int i = 0; i < OZ_SLOTS; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * i));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(empty0 + 8 * i));   // both issuers
    }
    for (int i = 0; i < OZ_ACC; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(accf0 + 8 * i));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(acce0 + 8 * i), "r"(OZ_EPI_WARPS));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(drain));
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

  if (warp == 0 && lane == 0) {
    // producer
    const uint32_t s0 = smem_u32(smem);
    uint32_t used = 0, eph = 0, fph = 0;   // slots loaded before; parity of the next empty wait and of the last load
    bool ok = true;
    for (long long t = blockIdx.x; t < total && ok && !s_err; t += gridDim.x) {
      int z, trow, tcol;
      if (!tile(t, z, trow, tcol)) continue;
      for (int part = 0; part < parts && ok; ++part) {
        // the previous panel's trailing block starts 128 rows and columns earlier
        const bool pv = part + 1 < parts;
        const unsigned char* ga = (pv ? prev.a : cur.a) + z * st.a + (long long)(trow + (pv ? 1 : 0)) * OZ_NCH * OZ_S * OZ_A;
        const unsigned char* gb = (pv ? prev.b : cur.b) + z * st.b + (long long)(tcol + (pv ? CW : 0)) * OZ_NCH * OZ_S * OZ_B;
        ok = oz_load_tile(std::make_integer_sequence<int, OZ_LOADS>{}, ga, gb, s0, full0, empty0, used, eph, fph);
      }
    }
    if (!ok) fail();
    // copies in flight land before the CTA can leave: the last load of each slot
    for (int q = 0; q < OZ_SLOTS; ++q)
      if ((used >> q) & 1) mbar_wait_suspend(full0 + 8 * q, (fph >> q) & 1);
  } else if (warp == 1 || warp == 2) {
    const uint32_t s0 = smem_u32(smem);
    const uint64_t da = umma_desc(s0, 128, OZ_ASBO), db = umma_desc(s0 + OZ_A, 128, OZ_BSBO);
    const bool issue = elect_one();
    OzSync sync{full0, acce0};
    bool ok = true;
    for (long long t = blockIdx.x; t < total && ok; t += gridDim.x) {
      if (__shfl_sync(0xffffffffu, s_err, 0)) break;
      int z, trow, tcol;
      if (!__shfl_sync(0xffffffffu, tile(t, z, trow, tcol), 0)) continue;
      auto plan = [&](auto pl) {
        using P = decltype(pl);
        return oz_run<P::p0>(tmem, da, db, issue, empty0, accf0, sync) &&
               oz_run<P::p1>(tmem, da, db, issue, empty0, accf0, sync) &&
               oz_run<P::p2>(tmem, da, db, issue, empty0, accf0, sync) &&
               oz_run<P::p3>(tmem, da, db, issue, empty0, accf0, sync);
      };
      for (int part = 0; part < parts && ok; ++part)
        ok = warp == 1 ? plan(OzPlan<OZ_WHO0>{}) : plan(OzPlan<OZ_WHO1>{});
    }
    if (!ok && issue) fail();
    // every MMA issued has completed before the tensor memory is freed
    if (issue)
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(drain) : "memory");
    __syncwarp();
    mbar_wait_suspend(drain, 0);
  } else if (warp >= 4) {
    // epilogue: thread = TMEM lane (row), OZ_EC complex columns of the tile
    const int lq = warp & 3, part_c = ((warp - 4) >> 2) * OZ_EC;
    const int row = lq * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)part_c;
    bool ok = true;
    int turn = 0;
    // exact powers of two: their reciprocals are a subtraction of exponents
    auto inverse = [](double x) { return __hiloint2double(0x7fe00000 - __double2hiint(x), 0); };
    for (long long t = blockIdx.x; t < total; t += gridDim.x) {
      int z, trow, tcol;
      if (!tile(t, z, trow, tcol)) continue;
      const int n = b.order(z);
      turn ^= 1;
      const long long zs = z * st.s;
      if (warp < 4 + OZ_N / 32) {
        const int j = (warp - 4) * 32 + lane;
        const double cc = cur.cb[zs + tcol * OZ_N + j];
        s_col[turn][0][j] = cc;
        if (parts > 1) s_col[turn][1][j] = prev.cb[zs + tcol * OZ_N + OZ_M + j] * inverse(cc);
      }
      const double rs = cur.ra[zs + trow * OZ_M + row];
      const double rr = parts > 1 ? prev.ra[zs + (trow + 1) * OZ_M + row] * inverse(rs) : 0.;
      // every epilogue thread: the scales are there, and nobody reads the tile before last's
      asm volatile("bar.sync 1, %0;" ::"n"(32 * OZ_EPI_WARPS) : "memory");
      ok = ok && !__shfl_sync(0xffffffffu, s_err, 0);
      if (!ok) continue;   // the others still meet at the barrier
      const int gr = r1 + trow * OZ_M + row, c0 = r1 + tcol * OZ_N + part_c;
      const int ncol = min(OZ_EC, n - c0);
      double2* C = b.sys(z) + gr + (long long)n * c0;
      // the tile comes into L2 while its products run
      if (gr < n && (lane & 7) == 0)
        for (int j = 0; j < ncol; ++j) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + (long long)n * j));
      double ar[OZ_EC], ai[OZ_EC];
#pragma unroll
      for (int j = 0; j < OZ_EC; ++j) ar[j] = ai[j] = 0.;
      // accumulator pairs: diagonals (7, 6), (5, 4) of the first phase pair, (0, 1), (2, 3)
      // of the second; the lighter diagonal is the odd one
#pragma unroll 1
      for (int pq = 0; pq < 4 * parts && ok; ++pq) {
        const int q = pq & 3;
        if (pq == 4) {
          // the deferred panel's sums in this panel's scales, exactly
#pragma unroll
          for (int j = 0; j < OZ_EC; ++j) {
            const double f = rr * s_col[turn][1][part_c + j];
            ar[j] *= f;
            ai[j] *= f;
          }
        }
        const int a0 = 2 * (q & 1);
        const bool got = mbar_wait_suspend(accf0 + 8 * a0, q >> 1) && mbar_wait_suspend(accf0 + 8 * (a0 + 1), q >> 1);
        if (!(ok = __all_sync(0xffffffffu, got))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t tlo = tl + (uint32_t)((q < 2 ? a0 : a0 + 1) * 2 * OZ_N);   // diagonals 7, 5, 1, 3
        const uint32_t thi = tl + (uint32_t)((q < 2 ? a0 + 1 : a0) * 2 * OZ_N);   // diagonals 6, 4, 0, 2
        // weight of the lighter diagonal, 256^(7 - s): 1, 2^16, 2^48, 2^32
        const double wt = __hiloint2double((1023 + (q < 2 ? 16 * q : 80 - 16 * q)) << 20, 0);
#pragma unroll
        for (int h = 0; h < 2 * OZ_EC / 8; ++h) {   // eight columns of Re, then of Im
          constexpr int HR = OZ_EC / 8;
          uint32_t lo[8], hi[8];
          const uint32_t off = (uint32_t)((h / HR) * OZ_N + (h % HR) * 8);
          tmem_ld8(tlo + off, lo);
          tmem_ld8(thi + off, hi);
          tmem_ld_wait(lo, hi);
          if (h == 2 * HR - 1) {   // both accumulators are read: release them
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acce0 + 8 * a0) : "memory");
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acce0 + 8 * (a0 + 1)) : "memory");
            }
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            // v = 256 hi + lo, |v| < 2^34, as the double 2^52 + 2^51 + 2^31 + v by its bits
            const long long bits = (long long)(int)hi[j] * 256 +
                                   (long long)(0x4338000000000000ull | (unsigned long long)(lo[j] ^ 0x80000000u));
            const double v = __longlong_as_double(bits) - 6755401588539392.;
            double& a = h < HR ? ar[8 * (h % HR) + j] : ai[8 * (h % HR) + j];
            a = fma(v, wt, a);
          }
        }
      }
      if (ok && gr < n) oz_subtract(C, n, ncol, rs, &s_col[turn][0][part_c], ar, ai);
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

// tiles of a full update of one system's trailing block
inline long long oz_tiles(int rest) {
  return (long long)((rest + OZ_M - 1) / OZ_M) * ((rest + OZ_N - 1) / OZ_N);
}

// The panel's trailing block from its images (and the deferred panel's in prev);
// corner: only what the next panel needs, its 128 columns and rows
inline void oz_apply(const OzSet& cur, const OzSet& prev, const OzStride& st, Batch b, int k0, int nsys,
                     cudaStream_t stream, long long& launches, int* status, bool corner) {
  const int rest = b.n - k0 - LU_OUTER;
  if (rest <= 0) return;
  const int nti = (rest + OZ_M - 1) / OZ_M, ntc = (rest + OZ_N - 1) / OZ_N;
  constexpr int CW = LU_OUTER / OZ_N;
  static std::atomic<unsigned long long> attr{0};
  static int sms = 0;
  once_per_device(attr, [] {
    cudaFuncSetAttribute(oz_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, OZ_SMEM);
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  });
  const long long tiles = corner ? (long long)(CW * nti + std::max(0, ntc - CW)) * nsys : oz_tiles(rest) * nsys;
  const int grid = (int)std::min<long long>(tiles, sms > 0 ? sms : 148);
  oz_update_kernel<<<grid, OZ_THREADS, OZ_SMEM, stream>>>(b, k0, cur, prev, st, nsys, status, nti, ntc, corner ? 1 : 0);
  ++launches;
}

}  // namespace nb200
