// The FP64 form's three contractions on the 5th-generation tensor cores by
// exact integer products (the Ozaki scheme: K. Ozaki, T. Ogita, S. Oishi,
// S. M. Rump, "Error-free transformations of matrix multiplication by using
// fast routines of matrix multiplication and its applications", Numer.
// Algorithms 59 (2012) 95-118):
//   T1   tmp_l  = B_l C5          (src/utils.jl:19-20, src/integrals.jl:150-152)
//   T2   b_pq^l = C5^T tmp_l
//   Y    Y      = sum_l tmp_l W_l  (the restructured Lagrangian of lagrange.cu)
//
// Digits.  T1's operands are seven signed 7-bit digits below a power of two,
//     x = 2^e sum_{i<7} d_i 2^(-7(i+1)),   d_i = trunc(128 r_i), r_(i+1) = 128 r_i - d_i,
// with 2^e the smallest power of two above the row's (column's) largest |x|.  The
// others are seven balanced 8-bit digits below any scale s, |x| <= F s (F = 0.498),
//     x = s sum_{i<7} d_i 256^-(i+1),   d_i in [-128, 127]:
// with the integer X = rint(x / s 2^56) the bytes of X + sum_i 128 256^i are d_i + 128,
// so one 64-bit addition yields every digit, and the residual is rounded to nearest.
//   b, C5 (T1)  truncated digits, one scale per row m of b_l (made once per job) and
//         per column q
//   C5 (T2)     balanced digits, one scale per column
//   tmp   balanced, scale RL[l] CN[q]: the largest row norm of b_l times the norm
//         of column q bounds |tmp_l[m, q]| (Cauchy-Schwarz), so the digits are
//         written by T1's epilogue with no pass for a maximum; the bound is 2-3
//         bits above the largest value
//   W     balanced digits of RL[l] CN[q] W_l[q, b], one scale per b (beta_b times the
//         largest |RL CN b_pq[b, q]| of that b, and the largest |RL CN t_b|, found by
//         T2's epilogue and the diagonal kernel), so that tmp's scales drop out of Y's
//         sum over (q, l)
// A product keeps the digit pairs with i + j < NG, NG = 7 in T1 and 8 in T2 and Y:
// exact s8 x s8 -> s32 sums (tcgen05.mma kind::i8) in NG TMEM accumulators (one per
// i + j, 64 columns each), combined in FP64 by the epilogue (exact int32 -> double,
// Horner in 2^-7 or 2^-8).  |sum| <= 7 * 2^14 * K < 2^31 for K <= 18688; Y's K range is
// cut accordingly.
// T1 is within 1e-13 of the FP64 product, row by row of b_l.  T2 and Y are, by the norm,
// as near to theirs as an FP64 GEMM (error of b_pq 1.4e-16 of the norm, of Y 2.1e-16, the
// GEMM's 3.3e-16 and 9.7e-16, nbf = 96, random b; NG = 7 left 1.6e-15 in Y).  The
// optimisers divide by gradient elements, so noise of 1e-14 in T2 and Y showed as 1e-8 in
// the orbitals.
//
// What is held in fixed point is relative to a bound of many elements: tmp to the largest
// row of b_l, column b of W to its largest term.  Elements far below lose bits that FP64
// would keep (three water molecules, orbitals of the core Hamiltonian: the median element
// of b_pq is off by 2.2e-12 of itself instead of 2.0e-12; J, K, Y and elag, sums over l,
// are not further off).  A row m of Y is as good as T1's noise (2^-44) allows while its
// largest row norm over l is within 2^6 of the largest of all rows: 2^-57 2^6 from tmp's
// digits, and as much again squared from W's where the orbitals are the basis functions
// themselves.  Molecules lie within that (water: 5).  A job whose rows spread further
// (ROW_SPREAD) keeps T1 from digits and takes T2 and Y as FP64 GEMMs: on rows 1e-9 and
// 1e6 times the others the digit products left nothing of the small rows.
//
// One persistent kernel, oz_kernel<MODE>, with TMEM accumulators of 64 columns each
// for a 128 x 64 output tile: warp 16 streams A's slices (16 KB TMA boxes, no
// multicast) through a ring, warp 17 issues the MMAs, warps 0-15 drain TMEM.
// B's slices are adjacent in shared memory, so the products of one A slice with
// several B slices are one MMA of N = 64 x (slices) <= 256.
//   T1: rows (m, l) flattened: no tile is cut at an aux index.  A = b's slices,
//       B = C5's.
//   T2: rows (q, l) flattened.  A = tmp's slices read MN-major, B = C5's.
//   Y:  rows m, K = (q, l).  A = the same slices of tmp read K-major, B = W's;
//       a unit is (tile, K range), its FP64 partial left for the tail to sum.
// T1 and T2 keep the C5 slices of the CTA's column tile in shared memory for the
// whole launch where they fit (nbf <= 256); a CTA then serves one column tile.
//
// Measured on one B200 (us; in brackets T1 alone from digits, T2 and Y as FP64 GEMMs):
//   nbf / naux / nbf5    T1            T2            W            Y            Lagrangian
//   256 / 1024 / 64      106 (131)     40 (85)       19 (20)      33 (81)      (orbital step 328 (434))
//   202 / 974 / 198      273 (470)     312 (761)     144 (186)    238 (841)    1094 (2235)
//   384 / 1856 / 320     1753 (2049)   1711 (4649)   548 (698)    1386 (6958)  6283 (14322)
// (in a loop, the larger two at the 1.74 GHz of the power cap).
// At nbf5 = 64 T1 is bound by HBM (b's slices in, tmp's out: 587 MB, 91 us at 6.45
// TB/s); the larger ones by what the MMAs and the TMA need of shared memory (a
// chunk of Y: 448 KB of operand reads, 168 KB written, 4900 cycles at 128 bytes a
// cycle; 5100 measured) and, in T1 and T2, by the drain between two rounds.
// elag is within 1e-15 of what the FP64 GEMMs make of the same tmp; its error against
// 64 bits, 7.2e-14 of the norm, is that of T1's truncated digits.
//
// Every wait is bounded; on a timeout the CTA records the failure in the
// context's failure word, drains its copies and MMAs, frees TMEM and exits.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <math.h>
#include <stdint.h>

#include <atomic>

#include "kernels.cuh"
#include "sm100.cuh"

namespace donof {

namespace oz {

constexpr int S = 7;                        // digits of every operand
constexpr int NG_MAX = 8;                   // accumulators: digit pairs with i + j < NG
constexpr double F = 0.498;                 // largest |x| / scale: every balanced digit fits [-128, 127]
constexpr double ROW_SPREAD = 64.0;         // largest ratio of b's row norms that T2 and Y take as digits
constexpr int EPI_WARPS = 16;               // four per TMEM lane quarter, 16 columns each (8 of 32: T1 148 against 113 us at nbf5 = 64)
constexpr int PRODUCER = EPI_WARPS;         // TMA producer
constexpr int ISSUER = EPI_WARPS + 1;       // TMEM allocator + MMA issuer
constexpr int NTHREADS = 32 * (EPI_WARPS + 2);
// 18 warps put 5 on one SM sub-partition of 16384 registers: at most 96 per thread
constexpr int BOUND_THREADS = 640;
constexpr int KC = 128;                     // K per stage: eight 16-byte groups of int8
constexpr int MT = 128;                     // rows per tile (MMA M)
constexpr int QT = 64;                      // columns per tile (MMA N per B slice)
constexpr int A_BYTES = MT * KC;            // 16 KB: one slice of A over (row tile, K chunk)
constexpr int BS_BYTES = QT * KC;           // 8 KB: one slice of B over (column tile, K chunk)
constexpr int RING_MAX = 8;                 // A stages in flight
constexpr int OFF_BAR = 0;
constexpr int OFF_MISC = 512;               // tmem base, abort flag
constexpr int OFF_DATA = 1024;              // B stages, then the A ring
constexpr int DATA_BYTES = 224 * 1024;
constexpr int SMEM_ALLOC = OFF_DATA + DATA_BYTES + 1024;  // slack for 1024-B alignment
static_assert(SMEM_ALLOC <= 227 * 1024, "shared memory budget");
static_assert(NG_MAX * QT <= 512, "TMEM columns");
constexpr int KMAX_CHUNKS = 146;            // 7 * 2^14 * 146 * 128 < 2^31
static_assert(7ll * 16384 * KMAX_CHUNKS * KC < (1ll << 31), "int32 accumulators");

// barrier indices
constexpr int A_FULL = 0;                   // +s (RING_MAX): A stage landed
constexpr int A_EMPTY = RING_MAX;           // +s: A stage consumed by the MMAs
constexpr int B_FULL = 2 * RING_MAX;        // +stage: B stage landed (resident: one per K chunk)
constexpr int B_STAGES = 8;
constexpr int B_EMPTY = B_FULL + B_STAGES;  // +slot (2): streamed B stage consumed
constexpr int ACC_FULL = B_EMPTY + 2;       // accumulators of a round complete: +0 the last, +1 those from 4 on, +2 3..0
constexpr int GFREE = ACC_FULL + 3;         // +g (NG_MAX): accumulator g drained and zeroed (count EPI_WARPS)
constexpr int B_END = GFREE + NG_MAX;       // every MMA of the CTA complete
static_assert((S * BS_BYTES) >> 4 == 4 * ((2 * 16 * S * QT) >> 4), "B stages adjoin");
static_assert((B_END + 1) * 8 <= OFF_MISC, "barrier area");

enum Mode {
    T1_DIGITS = 0,  // tmp as digit slices
    T1_F64 = 1,     // tmp in FP64
    T2 = 2,         // b_pq in FP64
    YSUM = 3,       // FP64 partials of Y
};

constexpr int accumulators(int mode) { return mode == T2 || mode == YSUM ? 8 : 7; }

struct Params {
    int nbf, nbf5, naux, ldq;  // ldq: nbf5 rounded up to 16 (row length of tmp's and W's slices per l)
    int nrt, nct;              // row tiles (128), column tiles (64)
    int nkc;                   // K chunks (128): all of T1's and T2's range, the whole (q, l) range for Y
    int cpu, nsplit;           // Y: chunks per unit, units per tile
    int k4_last;               // 32-wide K steps of the last chunk
    int resident;              // B's stages of the CTA's column tile are loaded once and kept
    int ring;                  // A stages
    int ring_off;              // byte offset of the ring behind OFF_DATA
    const double* sa;          // 2^ea per row (m, l) of b
    const double* RL;          // per l
    const double* RLi;         // per l: 1 / RL (0 for b_l = 0)
    const double* CN;          // per q
    const double* cb;          // per q: 2^(eb - 14) 2^56 / CN
    const double* sb1;         // per q: 2^(eb - 14), of C5's truncated digits
    const double* sb2;         // per q: s 2^-16, of its balanced digits
    const double* beta;        // per b (Y)
    unsigned *wm, *wt;         // per b: high words of the largest |RL CN b_pq[b, q]| (T2; null: not wanted) and |RL CN t_b|
    int8_t* t8;                // tmp's slices (see the layout above t8_at)
    double* out;               // FP64 output
    double* diag;              // T2: b_qq^l at q + nbf5 l
    int* fail;                 // the context's failure word for mbarrier waits
    long long wait;            // cycle budget of every bounded wait (drains excepted)
};

using namespace sm100;

// Exact int32 -> double: the bits 0x43300000:(x ^ 2^31) are the double
// 2^52 + 2^31 + x, from which 2^52 + 2^31 is subtracted exactly (an integer
// op and an FP64 add instead of a conversion-pipe instruction).
__device__ __forceinline__ double exact_f64(int x) {
    return __hiloint2double(0x43300000, x ^ (int)0x80000000) - 4503601774854144.0;
}

// Layout of the slices (the MMAs read them without swizzle): 128-wide chunks of the
// contiguous index (R = q + ldq l of tmp and W, n of b and C5), each in eight groups
// of 16, a group's 16 bytes contiguous and the rows one 16-byte step apart.
//   b    b8[n % 16 + 16 (r % 128 + 128 (n / 16 + ldn/16 (i + 7 (r / 128))))]   r = m + nbf l
//   tmp  t8[R % 16 + 16 (m + nbf (g + 8 (i + 7 chunk)))]      g = R / 16 % 8, chunk = R / 128
//   W    w8[R % 16 + 16 (b + nbf5 (j + 7 (g + 8 chunk)))]
//   C5   c8[n % 16 + 16 (q + nbf5 (j + 7 (g + 8 chunk)))]  (two: truncated and balanced)
// A row step of 16 bytes makes the stores contiguous over a warp's rows (512 bytes an
// instruction: with rows 128 bytes apart W's kernel took 185 instead of 126 us at
// nbf5 = 198), gives the 8 x 16-byte core matrices that a K-major and an MN-major
// operand share, and W's and C5's digits lie one after the other along N for every
// group.  A box is rows of 2 KB: T1's loads alone took 234 us at nbf = 202 as 128
// swizzled rows of 128 bytes at a pitch of 208, and take 160 us so.
__device__ __forceinline__ size_t t8_at(int R, int m, int nbf) {  // digit 0; digit i: + 128 nbf i
    return 16 * ((size_t)nbf * ((size_t)(R >> 7) * 8 * S + ((R >> 4) & 7)) + m) + (R & 15);
}

// The seven digits of z (|z| <= F 2^56) as bytes: byte 6 - i is digit i.
__device__ __forceinline__ unsigned long long digits7(double z) {
    const unsigned long long bias = 0x0080808080808080ull;
    return (unsigned long long)(__double2ll_rn(z) + (long long)bias) ^ bias;
}

// Byte transposition of four 7-byte digit strings: w[i] = digit i of z0, z1, z2, z3.
__device__ __forceinline__ void pack4(const unsigned long long (&z)[4], unsigned (&w)[S]) {
    const unsigned a0 = (unsigned)z[0], a1 = (unsigned)z[1], a2 = (unsigned)z[2], a3 = (unsigned)z[3];
    const unsigned h0 = (unsigned)(z[0] >> 32), h1 = (unsigned)(z[1] >> 32), h2 = (unsigned)(z[2] >> 32),
                   h3 = (unsigned)(z[3] >> 32);
    unsigned t0 = __byte_perm(a0, a1, 0x5140), t1 = __byte_perm(a2, a3, 0x5140);
    w[6] = __byte_perm(t0, t1, 0x5410);
    w[5] = __byte_perm(t0, t1, 0x7632);
    t0 = __byte_perm(a0, a1, 0x7362);
    t1 = __byte_perm(a2, a3, 0x7362);
    w[4] = __byte_perm(t0, t1, 0x5410);
    w[3] = __byte_perm(t0, t1, 0x7632);
    t0 = __byte_perm(h0, h1, 0x5140);
    t1 = __byte_perm(h2, h3, 0x5140);
    w[2] = __byte_perm(t0, t1, 0x5410);
    w[1] = __byte_perm(t0, t1, 0x7632);
    t0 = __byte_perm(h0, h1, 0x7362);
    t1 = __byte_perm(h2, h3, 0x7362);
    w[0] = __byte_perm(t0, t1, 0x5410);
}

// 32 bytes in one store (dst 32-byte aligned)
__device__ __forceinline__ void store_f64x4(double* dst, double a, double b, double c, double d) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(dst), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// |x| <= value_above(high word of |x|): the bits of the next high word (NaN for a
// NaN or an infinity).
__device__ __forceinline__ double value_above(unsigned hi) {
    return __hiloint2double((int)(hi < 0x7ff00000u ? hi + 1u : 0x7ff80000u), 0);
}

// The scale over F of the digits of W's column b: an upper bound of its largest
// |RL CN W| (NaN when a term was not finite); 0 when the column is zero.
__device__ __forceinline__ double w_scale(double beta, unsigned wm, unsigned wt) {
    const double s = (beta * value_above(wm) + value_above(wt)) * (1.0 + 0x1p-40);
    return s < 1e-290 ? 0.0 : s;
}

// The work of one CTA: unit u = (row tile, column tile, K range).
struct Unit {
    int row, col;  // tile indices
    int c0, nc;    // K chunks [c0, c0 + nc)
    int split;
};

template <int MODE, bool RES>
__device__ __forceinline__ int unit_count(const Params& P) {
    const int c = blockIdx.x, G = gridDim.x;
    if (MODE == YSUM) {
        const int n = P.nrt * P.nct * P.nsplit;
        return (n - c + G - 1) / G;
    }
    if (RES) {  // CTA c serves column tile c % nct, every (G of that tile)-th row tile
        const int ct = c % P.nct, gc = (G - ct + P.nct - 1) / P.nct, r0 = c / P.nct;
        return r0 < P.nrt ? (P.nrt - r0 + gc - 1) / gc : 0;
    }
    const int n = P.nrt * P.nct;
    return (n - c + G - 1) / G;
}

template <int MODE, bool RES>
__device__ __forceinline__ Unit unit_of(const Params& P, int u) {
    const int c = blockIdx.x, G = gridDim.x;
    Unit w;
    w.c0 = 0;
    w.nc = P.nkc;
    w.split = 0;
    if (MODE == YSUM) {
        const int i = c + u * G, tiles = P.nrt * P.nct;
        w.split = i / tiles;
        const int t = i - w.split * tiles;
        w.row = t % P.nrt;
        w.col = t / P.nrt;
        w.c0 = w.split * P.cpu;
        w.nc = min(P.cpu, P.nkc - w.c0);
    } else if (RES) {
        const int ct = c % P.nct, gc = (G - ct + P.nct - 1) / P.nct;
        w.row = c / P.nct + u * gc;
        w.col = ct;
    } else {
        const int i = c + u * G;
        w.row = i / P.nct;
        w.col = i - w.row * P.nct;
    }
    return w;
}

// One elected lane's MMAs of A slice i over NCH K chunks (A stages at descriptors ad,
// B stages one after the other from bd; the last chunk has nk4 steps of 32 K) with B
// slices 0 .. cnt-1: accumulators i .. i + cnt - 1, as one MMA of N = 64 cnt or two
// (7 = 4 + 3, 6 = 3 + 3, 5 = 3 + 2); part 1 the lower of the two, part 2 the upper, 3
// both.  With `commit`, `done` are the barriers that commits behind them arrive on.
// i and part are constants after unrolling.  The code is kept short as well as straight:
// it runs once a round beside 16 epilogue warps, and MMAs of 48 to 128 cycles take 100
// to issue there (46 in a loop of their own).  With a copy for every nk4 T2 took 322 and
// Y 246 us at nbf = 202 against 312 and 238.
template <int MODE, int NCH>
__device__ __forceinline__ void issue_slice(int i, int part, uint32_t tmem, const uint64_t (&ad)[NCH], uint64_t bd,
                                            int nk4, const uint32_t (&done)[NCH], bool commit) {
    constexpr int NG = accumulators(MODE);
    const int cnt = (NG - i) < S ? (NG - i) : S;
    const int first = cnt <= 4 ? cnt : (cnt + 1) / 2;
    // 32 K further: two groups, or for the MN-major operand four 8-row core matrices
    constexpr uint64_t astep = (MODE == T2 ? 32 * 16 : 2 * 16 * MT) >> 4;
    constexpr uint64_t bstep = (2 * 16 * S * QT) >> 4;
    constexpr uint32_t amn = MODE == T2 ? 1u << 15 : 0u;
    auto step = [&](uint64_t a, uint64_t b) {
        if (part & 1) umma_i8(tmem + (uint32_t)(i * QT), a, b, idesc_i8(MT, QT * first) | amn, 1u);
        if ((part & 2) && cnt > first)
            umma_i8(tmem + (uint32_t)((i + first) * QT), a, b + (uint64_t)(first * QT),
                    idesc_i8(MT, QT * (cnt - first)) | amn, 1u);
    };
    if (elect_one()) {
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
            const uint64_t a = ad[c], b = bd + (uint64_t)c * (4 * bstep);
            const int n = c == NCH - 1 ? nk4 : KC / 32;
            if (c < NCH - 1) {
#pragma unroll
                for (int k4 = 0; k4 < KC / 32; ++k4) step(a + k4 * astep, b + k4 * bstep);
            } else {
                step(a, b);
                if (n > 1) step(a + astep, b + bstep);
                if (n > 2) step(a + 2 * astep, b + 2 * bstep);
                if (n > 3) step(a + 3 * astep, b + 3 * bstep);
            }
        }
        if (commit) {
#pragma unroll
            for (int c = 0; c < NCH; ++c) umma_commit(done[c]);
        }
    }
    __syncwarp();
}

// Descriptors of an A stage and of a B stage.
template <int MODE>
__device__ __forceinline__ uint64_t a_desc(uint32_t addr) {
    if (MODE == T2) return sdesc_flat(addr, 128, 16 * MT);  // MN-major: (q, l) along M, 8 m per 128 bytes
    return sdesc_flat(addr, 16 * MT, 128);                  // K-major: groups of 16 K 2 KB apart
}
__device__ __forceinline__ uint64_t b_desc(uint32_t addr) {
    return sdesc_flat(addr, 16 * S * QT, 128);
}

// Round r of a CTA = one unit: its MMAs accumulate into the NG accumulators, then
// the epilogue drains them.  A's slices are consumed from the least significant
// (i = 6) to the most: slice i writes accumulators i .. i + 6 only, so the first
// MMAs of round r + 1 need only the top accumulators, which the epilogue of round
// r drains (and zeroes) first.  The drain of accumulator g is a TMEM load and a
// store of zeros; its release (GFREE[g]) comes right after, and the FP64
// arithmetic of the epilogue runs while the next round's MMAs already fill the
// released columns.
// A round ends with slice 0 against B's upper slices (accumulators 6..4), then its
// lower ones (3..0): accumulator 7 (NG = 8) is complete a slice earlier, 6..4 half a
// slice earlier, so the epilogue drains them while the last MMAs run and the tensor
// cores do not wait for it between rounds.  With B resident (NKC = its K chunks, 1 or
// 2) the order is slice-major over the K chunks and a slice's MMAs of both chunks are
// one block of the elected lane (T1 at nbf = 256: 111 us, 118 chunk by chunk); with B streamed
// (NKC = 0) it is chunk by chunk.
template <int MODE, int NKC>
__global__ void __launch_bounds__(BOUND_THREADS, 1)
oz_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Params P) {
    constexpr int NG = accumulators(MODE);
    constexpr int B_BYTES = S * BS_BYTES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t sbase = saddr(sm) + OFF_DATA;
    const uint32_t sring = sbase + (uint32_t)P.ring_off;
    const uint32_t sbar = saddr(sm) + OFF_BAR;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(sm + OFF_MISC);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + OFF_MISC + 16);
    auto bar = [&](int i) { return sbar + 8u * (uint32_t)i; };
    auto wait_on = [&](uint32_t b, uint32_t parity) {  // of a whole warp
        bool r = mbar_try(b, parity);
        if (!__all_sync(0xffffffffu, r)) r = mbar_wait(b, parity, abort_flag, P.wait);
        return __all_sync(0xffffffffu, r) != 0;
    };
    auto wait = [&](int i, uint32_t parity) { return wait_on(bar(i), parity); };

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    constexpr bool resident = NKC > 0;
    const int my_units = unit_count<MODE, resident>(P);

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i <= B_END; ++i) mbar_init(bar(i), (i >= GFREE && i < GFREE + NG_MAX) ? EPI_WARPS : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == ISSUER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(saddr(tmem_slot)));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == PRODUCER) {
        // ------------------------------------------------------------ producer
        // Every lane of the warp waits, one elected lane issues (a wait by lane 0
        // alone, broadcast to the others, took 560 cycles a stage instead of 75).
        if (my_units > 0) {
            int it = 0, s = 0, bs = 0;  // A stages issued, their slot, B stages issued
            uint32_t ph = 1;            // parity of the slot's "consumed" phase
            bool ok = true;
            auto load_a = [&](int i, int kc, int row) {
                if (!wait(A_EMPTY + s, ph)) return false;
                if (elect_one()) {
                    mbar_expect_tx(bar(A_FULL + s), (uint32_t)A_BYTES);
                    if (MODE == T2)  // 128 m (K) of the 128 (q, l) of a row tile
                        tma_load_3d(sring + s * A_BYTES, &map_a, bar(A_FULL + s), 2 * kc * KC, 0, i + S * row);
                    else if (MODE == YSUM)  // 128 (q, l) (K) of 128 m
                        tma_load_3d(sring + s * A_BYTES, &map_a, bar(A_FULL + s), 2 * row * MT, 0, i + S * kc);
                    else  // 128 n (K) of 128 (m, l)
                        tma_load_3d(sring + s * A_BYTES, &map_a, bar(A_FULL + s), 0, 8 * kc, i + S * row);
                }
                __syncwarp();
                ++it;
                if (++s == P.ring) {
                    s = 0;
                    ph ^= 1u;
                }
                return true;
            };
            auto load_b = [&](int stage, int col, int kc) {
                if (elect_one()) {
                    mbar_expect_tx(bar(B_FULL + stage), (uint32_t)B_BYTES);
                    tma_load_3d(sbase + stage * B_BYTES, &map_b, bar(B_FULL + stage), 2 * col * QT, 0, 8 * kc);
                }
                __syncwarp();
            };
            if (resident) {
                const int col = unit_of<MODE, resident>(P, 0).col;
                for (int kc = 0; kc < P.nkc; ++kc) load_b(kc, col, kc);
            }
            for (int u = 0; u < my_units && ok; ++u) {
                const Unit w = unit_of<MODE, resident>(P, u);
                if (resident) {
                    for (int i = S - 1; i >= 0 && ok; --i)
                        for (int kc = 0; kc < w.nc && ok; ++kc) ok = load_a(i, kc, w.row);
                    continue;
                }
                for (int kc = w.c0; kc < w.c0 + w.nc && ok; ++kc, ++bs) {
                    const int slot = bs & 1;
                    if (!wait(B_EMPTY + slot, (uint32_t)(((bs >> 1) & 1) ^ 1))) {
                        ok = false;
                        break;
                    }
                    load_b(slot, w.col, kc);
                    for (int i = S - 1; i >= 0 && ok; --i) ok = load_a(i, kc, w.row);
                }
            }
            // drain: every issued copy has landed before the CTA exits
            for (int j = (it > P.ring ? it - P.ring : 0); j < it; ++j)
                mbar_drain(bar(A_FULL + j % P.ring), (uint32_t)((j / P.ring) & 1));
            if (resident) {
                for (int kc = 0; kc < P.nkc; ++kc) mbar_drain(bar(B_FULL + kc), 0);
            } else {
                for (int j = (bs > 2 ? bs - 2 : 0); j < bs; ++j)
                    mbar_drain(bar(B_FULL + (j & 1)), (uint32_t)((j >> 1) & 1));
            }
        }
    } else if (warp == ISSUER) {
        // ------------------------------------------------------------ MMA issuer
        // accumulator g (TMEM columns [64 g, 64 g + 64)) collects D_i E_j, i + j = g.
        // The B slices lie one after the other in shared memory (slice j = rows
        // [64 j, 64 j + 64) of the stage), so D_i times slices j0 .. j0+c-1 is ONE
        // MMA with N = 64 c whose columns land on accumulators i+j0 .. i+j0+c-1.
        // The epilogue zeroes every accumulator it releases: all MMAs accumulate.
        // The whole warp runs the loop, one elected lane issues.
        if (my_units > 0) {
            // ring position: the full barrier and descriptor of the next stage, what is
            // left of the pass, its phase; the empty barriers lie RING_MAX behind
            uint32_t fb = bar(A_FULL), aph = 0;
            uint64_t ad = a_desc<MODE>(sring);
            int left = P.ring, bs = 0;
            bool ok = true;
            bool ready = false;  // this lane saw the next A stage land
            bool gready = false; // ... and the next accumulator released
            auto next = [&]() {  // to the next stage, whose arrival is asked for while MMAs are issued
                fb += 8u;
                ad += A_BYTES >> 4;
                if (--left == 0) {
                    fb = bar(A_FULL);
                    ad = a_desc<MODE>(sring);
                    left = P.ring;
                    aph ^= 1u;
                }
                ready = mbar_test(fb, aph);
            };
            auto landed = [&]() {
                if (!__all_sync(0xffffffffu, ready) && !wait_on(fb, aph)) return false;
                return true;
            };
            for (int u = 0; u < my_units && ok; ++u) {
                const uint32_t up = (uint32_t)(u & 1);
                if constexpr (resident) {
                    if (u == 0)
#pragma unroll
                        for (int kc = 0; kc < NKC; ++kc) ok = ok && wait(B_FULL + kc, 0);
#pragma unroll
                    for (int ii = 0; ii < S; ++ii) {
                        const int i = S - 1 - ii;
                        if (ii == 0)
                            for (int g = NG - 1; g >= i; --g) ok = ok && wait(GFREE + g, up);
                        else if (!__all_sync(0xffffffffu, gready))
                            ok = ok && wait(GFREE + i, up);
                        uint32_t done[NKC];
                        uint64_t da[NKC];
#pragma unroll
                        for (int kc = 0; kc < NKC; ++kc) {
                            ok = ok && landed();
                            if (!ok) break;
                            done[kc] = fb + 8u * RING_MAX;
                            da[kc] = ad;
                            next();
                        }
                        if (!ok) break;
                        if (i > 0) gready = mbar_test(bar(GFREE + i - 1), up);
                        fence_after();
                        issue_slice<MODE, NKC>(i, i > 0 ? 3 : 2, tmem, da, b_desc(sbase), P.k4_last, done, i > 0);
                        if (i == NG - S) {  // slice 1 (NG = 8) or the upper part of slice 0: the last accumulator
                            if (elect_one()) umma_commit(bar(ACC_FULL));
                            __syncwarp();
                        }
                        if (i == 0) {
                            if (elect_one()) umma_commit(bar(ACC_FULL + 1));
                            __syncwarp();
                            issue_slice<MODE, NKC>(0, 1, tmem, da, b_desc(sbase), P.k4_last, done, true);
                            if (elect_one()) umma_commit(bar(ACC_FULL + 2));
                            __syncwarp();
                        }
                    }
                } else {
                    const Unit w = unit_of<MODE, resident>(P, u);
                    const int end = w.c0 + w.nc;
                    for (int kc = w.c0; kc < end && ok; ++kc, ++bs) {
                        const int slot = bs & 1;
                        const uint64_t bd = b_desc(sbase + slot * B_BYTES);
                        const int nk4 = kc == P.nkc - 1 ? P.k4_last : KC / 32;
                        ok = wait(B_FULL + slot, (uint32_t)((bs >> 1) & 1));
#pragma unroll
                        for (int ii = 0; ii < S; ++ii) {
                            const int i = S - 1 - ii;
                            if (kc == w.c0)
                                for (int g = ii == 0 ? NG - 1 : i; g >= i; --g) ok = ok && wait(GFREE + g, up);
                            ok = ok && landed();
                            if (!ok) break;
                            const uint32_t done[1] = {fb + 8u * RING_MAX};
                            const uint64_t da[1] = {ad};
                            next();
                            fence_after();
                            if (i == 0 && kc == end - 1) {
                                issue_slice<MODE, 1>(0, 2, tmem, da, bd, nk4, done, false);
                                if (elect_one()) {
                                    if (NG == S) umma_commit(bar(ACC_FULL));
                                    umma_commit(bar(ACC_FULL + 1));
                                }
                                __syncwarp();
                                issue_slice<MODE, 1>(0, 1, tmem, da, bd, nk4, done, true);
                                if (elect_one()) umma_commit(bar(ACC_FULL + 2));
                                __syncwarp();
                            } else {
                                issue_slice<MODE, 1>(i, 3, tmem, da, bd, nk4, done, true);
                                if (NG > S && i == NG - S && kc == end - 1) {
                                    if (elect_one()) umma_commit(bar(ACC_FULL));
                                    __syncwarp();
                                }
                            }
                        }
                        if (ok && elect_one()) umma_commit(bar(B_EMPTY + slot));
                        __syncwarp();
                    }
                }
            }
            if (elect_one()) umma_commit(bar(B_END));
            __syncwarp();
            mbar_drain(bar(B_END), 0);  // every MMA of this CTA has completed
        }
    } else {
        // ------------------------------------------------------------ epilogue (warps 0-15)
        // warp w reads TMEM lanes [32 (w % 4), +32) = rows 128 row + 32 (w % 4) + lane,
        // and columns [16 (w / 4), +16) of every accumulator
        constexpr int NC = QT / 4;
        const int quarter = warp & 3, group = warp >> 2;
        const uint32_t tl = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(group * NC);
        // zero every accumulator and release it for the first round
#pragma unroll
        for (int g = 0; g < NG; ++g) tmem_zero16(tl + (uint32_t)(g * QT));
        tmem_wait_st();
        fence_before();
        __syncwarp();
        if (lane == 0)
            for (int g = 0; g < NG; ++g) mbar_arrive(bar(GFREE + g));
        unsigned top = 0;  // T2: largest high word of |RL CN b_pq| in column `group NC + lane` of the tile
        auto keep_top = [&](int q) {  // (lanes from NC on hold 0)
            if (lane < NC && q + lane < P.nbf5) atomicMax(P.wm + q + lane, top);
            top = 0;
        };
        for (int u = 0; u < my_units; ++u) {
            const Unit w = unit_of<MODE, resident>(P, u);
            const int R = w.row * MT + quarter * 32 + lane;
            const int q0 = w.col * QT + group * NC;
            // per-row data, read before the wait
            int l = 0, x = 0;  // aux index, and m (T1) or q (T2)
            bool in;
            double rs = 0.0;
            if (MODE == YSUM) {
                x = R;
                in = R < P.nbf;
            } else if (MODE == T2) {
                l = R / P.ldq;
                x = R - l * P.ldq;
                in = l < P.naux && x < P.nbf5;
                if (in) rs = P.RL[l] * P.CN[x];
            } else {
                l = R / P.nbf;
                x = R - l * P.nbf;
                in = l < P.naux;
                if (in) rs = MODE == T1_F64 ? P.sa[R] : P.sa[R] * P.RLi[l];
            }
            // Horner from the least significant accumulator: v = sum_g acc_g 2^(-8g), or 2^(-7g)
            constexpr double radix = MODE == T2 || MODE == YSUM ? 0x1p-8 : 0x1p-7;
            double v[NC];
            bool ok = true;
#pragma unroll
            for (int g = NG - 1; g >= 0; --g) {
                if (g == NG - 1 || g == NG - 2 || g == 3) {
                    ok = ok && wait(ACC_FULL + (g == NG - 1 ? 0 : g == NG - 2 ? 1 : 2), (uint32_t)(u & 1));
                    if (!ok) break;
                    fence_after();
                }
                uint32_t a[NC];
                tmem_issue16(tl + (uint32_t)(g * QT), a);
                tmem_wait_ld();
                tmem_zero16(tl + (uint32_t)(g * QT));
                tmem_wait_st();
                fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(GFREE + g));
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    const double t = exact_f64((int)a[k]);
                    v[k] = (g == NG - 1) ? t : fma(v[k], radix, t);
                }
            }
            if (!ok) break;
            if (MODE == T1_DIGITS) {
                // digit slices of tmp, q contiguous: 16 bytes per slice and thread; the
                // padding columns [nbf5, ldq) get cb = 0, i.e. zero digits
                unsigned wd[4][S];
#pragma unroll
                for (int k4 = 0; k4 < 4; ++k4) {
                    unsigned long long z[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) z[k] = digits7(v[4 * k4 + k] * (rs * P.cb[q0 + 4 * k4 + k]));
                    pack4(z, wd[k4]);
                }
                if (in && q0 < P.ldq) {
                    int8_t* dst = P.t8 + t8_at(P.ldq * l + q0, x, P.nbf);
#pragma unroll
                    for (int i = 0; i < S; ++i)
                        *reinterpret_cast<uint4*>(dst + (size_t)i * P.nbf * 128) =
                            make_uint4(wd[0][i], wd[1][i], wd[2][i], wd[3][i]);
                }
            } else if (MODE == T1_F64) {
                double* dst = P.out + (size_t)P.nbf * P.nbf5 * l + x;
#pragma unroll
                for (int k = 0; k < NC; ++k)
                    if (in && q0 + k < P.nbf5) dst[(size_t)P.nbf * (q0 + k)] = v[k] * rs * P.sb1[q0 + k];
            } else if (MODE == T2) {
#pragma unroll
                for (int k = 0; k < NC; ++k)
                    v[k] = v[k] * rs * P.sb2[q0 + k];  // b_pq (columns at and beyond nbf5: sb2 = 0)
                if (P.wm != nullptr) {
#pragma unroll
                    for (int k = 0; k < NC; ++k) {
                        const unsigned h = __reduce_max_sync(
                            0xffffffffu, in ? (unsigned)__double2hiint(v[k] * rs) & 0x7fffffffu : 0u);
                        if (lane == k) top = max(top, h);
                    }
                    if (!resident || u == my_units - 1) keep_top(q0);
                }
                if (in && x >= q0 && x < q0 + NC) {
                    double t = 0.0;
#pragma unroll
                    for (int k = 0; k < NC; ++k) t = q0 + k == x ? v[k] : t;
                    P.diag[x + (size_t)P.nbf5 * l] = t;
                }
                double* dst = P.out + ((size_t)P.nbf5 * l + x) * P.nbf5 + q0;
                if (in && q0 + NC <= P.nbf5 && (P.nbf5 & 3) == 0) {
#pragma unroll
                    for (int k = 0; k < NC; k += 4) store_f64x4(dst + k, v[k], v[k + 1], v[k + 2], v[k + 3]);
                } else if (in && q0 + NC <= P.nbf5 && (P.nbf5 & 1) == 0) {
#pragma unroll
                    for (int k = 0; k < NC; k += 2) *reinterpret_cast<double2*>(dst + k) = make_double2(v[k], v[k + 1]);
                } else if (in) {
#pragma unroll
                    for (int k = 0; k < NC; ++k)
                        if (q0 + k < P.nbf5) dst[k] = v[k];
                }
            } else {
                double* dst = P.out + (size_t)w.split * P.nbf * P.nbf5 + x;
#pragma unroll
                for (int k = 0; k < NC; ++k)
                    if (in && q0 + k < P.nbf5)
                        dst[(size_t)P.nbf * (q0 + k)] = v[k] * (w_scale(P.beta[q0 + k], P.wm[q0 + k], P.wt[q0 + k]) * (0x1p-16 / F));
            }
        }
    }

    fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag && P.fail) *reinterpret_cast<volatile int*>(P.fail) = 1;
    if (warp == ISSUER) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
    }
}

// ---------------------------------------------------------------- digit slices
// The seven balanced digits of x / s (|x| <= F s) as bytes: byte 6 - i is digit i.
__device__ __forceinline__ unsigned long long digits7(double x, double s) { return digits7(x / s * 0x1p56); }

// The seven truncated digits of y, |y| < 1: d_i = trunc(128 r_i), r_(i+1) = 128 r_i - d_i.
__device__ __forceinline__ unsigned long long truncated7(double y) {
    unsigned long long z = 0;
#pragma unroll
    for (int i = 0; i < S; ++i) {
        y *= 128.0;
        const double t = trunc(y);
        z = z << 8 | (unsigned)((int)t & 255);
        y -= t;
    }
    return z;
}

// The scale of balanced digits of a column whose largest |x| is mx (floored, so that
// x / s never overflows; a zero column has zero digits whatever its scale).
__device__ __forceinline__ double digit_scale(double mx) { return fmax(mx, 1e-280) / F; }

// Per row (m, l) of b: sa = 2^e with max_n |b| < 2^e (1 for a zero row), and the row
// norm's maxima over m into rn[l] and over l into rm[m] (bits of a non-negative double).
// One thread per (m, l), coalesced over m.
__global__ void row_scale_kernel(const double* __restrict__ b, int nbf, long long naux, double* __restrict__ sa,
                                 unsigned long long* __restrict__ rn, unsigned long long* __restrict__ rm) {
    const long long total = (long long)nbf * naux;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long l = i / nbf;
        const int m = (int)(i - l * nbf);
        const double* row = b + (long long)nbf * nbf * l + m;
        double mx = 0.0, ss = 0.0;
        for (int n = 0; n < nbf; ++n) {
            const double x = fabs(row[(long long)nbf * n]);
            mx = fmax(mx, x);
            ss += x * x;
        }
        double norm = sqrt(ss);
        if (mx > 0.0 && !(ss > 1e-250 && ss < 1e250)) {  // squares out of range: scaled by the maximum
            ss = 0.0;
            for (int n = 0; n < nbf; ++n) {
                const double x = row[(long long)nbf * n] / mx;
                ss += x * x;
            }
            norm = mx * sqrt(ss);
        }
        int e = 0;
        if (mx > 0.0) frexp(mx, &e);  // mx = f 2^e, f in [0.5, 1)
        sa[i] = isnan(norm) || isinf(mx) ? __longlong_as_double(0x7ff8000000000000ll) : ldexp(1.0, e);
        atomicMax(rn + l, (unsigned long long)__double_as_longlong(norm));
        atomicMax(rm + m, (unsigned long long)__double_as_longlong(norm));
    }
}

// The largest of rm[0 .. nbf) and the smallest that is not zero (infinity if all are), by
// one warp.
__global__ void row_spread_kernel(const double* __restrict__ rm, int nbf, double* __restrict__ out) {
    const double inf = __longlong_as_double(0x7ff0000000000000ll);
    double hi = 0.0, lo = inf;
#pragma unroll 4
    for (int m = threadIdx.x; m < nbf; m += 32) {
        const double x = rm[m];
        hi = fmax(hi, x);
        lo = fmin(lo, x > 0.0 ? x : inf);
    }
    for (int o = 16; o > 0; o >>= 1) {
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    }
    if (threadIdx.x == 0) {
        out[0] = hi;
        out[1] = lo;
    }
}

// rn[l] (bits) -> RL[l] = norm (1 + 2^-30) / F, RLi = 1 / RL in rn's place
__global__ void row_finish_kernel(long long naux, double* __restrict__ RL, double* __restrict__ rn) {
    for (long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x; l < naux;
         l += (long long)gridDim.x * blockDim.x) {
        double R = rn[l] * (1.0 + 0x1p-30) / F;
        if (R > 0.0 && R < 1e-290) R = 1e-290;  // 1 / R stays finite
        RL[l] = R;                              // NaN where b_l holds one: b_pq and Y follow
        rn[l] = R > 0.0 ? 1.0 / R : 0.0;
    }
}

// b's slices (layout above t8_at), n < ldn = nbf rounded up to 16.  32 x 32 (m, n)
// tiles through shared memory: reads coalesced over m, four n of one digit a 4-byte
// word.
__global__ void __launch_bounds__(256) split_b_kernel(const double* __restrict__ b, const double* __restrict__ sa,
                                                      int nbf, int ldn, long long naux, int8_t* __restrict__ out) {
    __shared__ double tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int tn = (nbf + 31) / 32;
    const long long tiles = (long long)tn * tn * naux;
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        const long long l = t / ((long long)tn * tn);
        const int r = (int)(t - l * tn * tn);
        const int m0 = 32 * (r % tn), n0 = 32 * (r / tn);
        const double* B = b + (long long)nbf * nbf * l;
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int m = m0 + tx, n = n0 + ty + 8 * k;
            tile[ty + 8 * k][tx] = (m < nbf && n < nbf) ? B[m + (long long)nbf * n] : 0.0;  // tile[n][m]
        }
        __syncthreads();
        // a warp: 8 m of 4 words (16 n)
        const int m = m0 + (ty & 3) * 8 + (tx >> 2), nq = 16 * (ty >> 2) + 4 * (tx & 3);
        if (m < nbf && n0 + nq < ldn) {  // ldn is a multiple of 16: whole words
            const double s = sa[m + (long long)nbf * l];
            unsigned long long z[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) z[k] = truncated7(tile[nq + k][m - m0] / s);
            unsigned w[S];
            pack4(z, w);
            const long long row = m + (long long)nbf * l;
            int8_t* dst = out + 16 * ((row & 127) + 128 * (((n0 + nq) >> 4) + (long long)(ldn / 16) * S * (row >> 7))) + (nq & 15);
#pragma unroll
            for (int i = 0; i < S; ++i) *reinterpret_cast<unsigned*>(dst + 128ll * ldn * i) = w[i];
        }
    }
}

struct PrepArgs {
    const double* C;
    const double *n, *cj12, *ck12;  // null: no W will be built
    int nbf, nbf5, nkc;             // grid: the columns rounded up to whole tiles
    double *sb1, *sb2, *CN, *cb, *beta;
    int8_t *c1, *c2;                // c8 of T1 and of T2, n padded to whole chunks with zeros
    unsigned *wm, *wt;              // zeroed
};

// One block per column q of C5 (and per padding column): both sets of digit slices, the
// scales of T1 and T2, and beta_q = the largest |factor| of W's column q.
__global__ void __launch_bounds__(128) prep_kernel(const PrepArgs a) {
    __shared__ double red[3][4];
    __shared__ double bc[3];
    const int q = blockIdx.x, tid = threadIdx.x;
    if (tid == 0) a.wm[q] = a.wt[q] = 0;
    if (q >= a.nbf5) {
        if (tid == 0) a.sb1[q] = a.sb2[q] = a.CN[q] = a.cb[q] = a.beta[q] = 0.0;
        return;
    }
    const double* col = a.C + (long long)a.nbf * q;
    double mx = 0.0, be = 0.0;
    for (int n = tid; n < a.nbf; n += blockDim.x) mx = fmax(mx, fabs(col[n]));
    bool bad = false;
    if (a.n != nullptr) {
        for (int p = tid; p < a.nbf5; p += blockDim.x) {
            const double x = a.cj12[q + (long long)a.nbf5 * p], y = a.ck12[q + (long long)a.nbf5 * p];
            be = fmax(be, fmax(fabs(x), fabs(y)));
            bad = bad || isnan(x) || isnan(y);
        }
        const double x = a.n[q];
        be = fmax(be, fabs(x));
        bad = bad || isnan(x);
    }
    auto reduce = [&](double x, int k, bool sum) {
        for (int o = 16; o > 0; o >>= 1) {
            const double y = __shfl_xor_sync(0xffffffffu, x, o);
            x = sum ? x + y : fmax(x, y);
        }
        if ((tid & 31) == 0) red[k][tid >> 5] = x;
        __syncthreads();
        if (tid == 0) {
            double t = red[k][0];
            for (int w = 1; w < 4; ++w) t = sum ? t + red[k][w] : fmax(t, red[k][w]);
            bc[k] = t;
        }
        __syncthreads();
        return bc[k];
    };
    mx = reduce(mx, 0, false);
    be = reduce(be, 1, false);
    const bool anybad = __syncthreads_or(bad);
    const double s = digit_scale(mx);
    int e = 0;
    if (mx > 0.0) frexp(mx, &e);
    const double inv = ldexp(1.0, -e);
    double ss = 0.0;
    for (int n = tid; n < a.nbf; n += blockDim.x) {
        const double x = col[n] / s;
        ss += x * x;
    }
    ss = reduce(ss, 2, true);
    if (tid == 0) {
        const double nan = __longlong_as_double(0x7ff8000000000000ll);
        double cn = s * sqrt(ss) * (1.0 + 0x1p-40);
        if (!isfinite(ss) || isinf(mx)) cn = nan;  // a column with a NaN or an infinity: every product of it is NaN
        a.CN[q] = cn;
        a.sb1[q] = isnan(cn) ? nan : ldexp(1.0, e - 14);  // 2^-14: the weight of digit pair (0, 0)
        a.sb2[q] = isnan(cn) ? nan : s * 0x1p-16;
        a.cb[q] = cn == 0.0 ? 0.0 : ldexp(1.0, e - 14) * 0x1p56 / cn;
        a.beta[q] = anybad ? nan : be;
    }
    for (int n = tid; n < a.nkc * KC; n += blockDim.x) {
        const double x = n < a.nbf ? col[n] : 0.0;
        const unsigned long long z1 = truncated7(x * inv), z2 = digits7(x, s);
        const long long at = (n & 15) + 16 * (q + (long long)a.nbf5 * S * (n >> 4));
#pragma unroll
        for (int i = 0; i < S; ++i) {
            a.c1[at + 16ll * a.nbf5 * i] = (int8_t)(z1 >> (8 * (S - 1 - i)));
            a.c2[at + 16ll * a.nbf5 * i] = (int8_t)(z2 >> (8 * (S - 1 - i)));
        }
    }
}

// ---------------------------------------------------------------- W
// tv[b + nbf5 l] = n'_b d_b^l + sum_q cj12[b, q] d_q^l with d_q^l = b_pq^l[q, q]
// (lagrange.cu), and the largest |RL CN tv| per b.  A block takes 32 b of LB aux
// indices: the diagonals (D, written by T2) staged in shared memory a panel of DQ at a time, each of
// its eight warps on an eighth of the panel's q (one cj12 element, read along b,
// serves LB products), the eight partial sums added in a fixed order.
constexpr int LB = 8;
constexpr int DQ = 256;

__global__ void __launch_bounds__(256) diag_kernel(const double* __restrict__ D, const double* __restrict__ n,
                                                   const double* __restrict__ cj12, int nbf5, int naux, int nalpha,
                                                   int nbeta, const double* __restrict__ RL,
                                                   const double* __restrict__ CN, double* __restrict__ tv,
                                                   unsigned* __restrict__ wt, unsigned* tail_words) {
    zero_tail_state(tail_words);
    __shared__ double sd[LB][DQ];
    __shared__ double part[8][LB][32];   // [warp][l][b]
    __shared__ unsigned tops[LB][32];    // [l][b]
    const int l0 = blockIdx.x * LB, b = blockIdx.y * 32 + (threadIdx.x & 31), warp = threadIdx.x >> 5;
    double s[LB];
#pragma unroll
    for (int k = 0; k < LB; ++k) s[k] = 0.0;
    for (int p0 = 0; p0 < nbf5; p0 += DQ) {
        const int np = min(DQ, nbf5 - p0);
        __syncthreads();
        if (l0 + warp < naux)  // warp k stages aux index l0 + k
            for (int q = threadIdx.x & 31; q < np; q += 32) sd[warp][q] = D[(size_t)nbf5 * (l0 + warp) + p0 + q];
        __syncthreads();
        if (b < nbf5) {
#pragma unroll 8
            for (int q = warp; q < np; q += 8) {
                const double c = cj12[b + (long long)nbf5 * (p0 + q)];
#pragma unroll
                for (int k = 0; k < LB; ++k) s[k] = fma(c, sd[k][q], s[k]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < LB; ++k) part[warp][k][threadIdx.x & 31] = s[k];
    __syncthreads();
    unsigned top = 0;
    const int l = l0 + warp;  // warp k finishes aux index l0 + k (LB warps)
    if (b < nbf5 && l < naux) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += part[w][warp][threadIdx.x & 31];
        const bool dj = (nbeta > 0) && (b < nbeta || b >= nalpha);
        if (dj) t = fma(n[b], D[(size_t)nbf5 * l + b], t);
        tv[b + (long long)nbf5 * l] = t;
        top = (unsigned)__double2hiint(RL[l] * t * CN[b]) & 0x7fffffffu;
    }
    tops[warp][threadIdx.x & 31] = top;
    __syncthreads();
    if (warp != 0 || b >= nbf5) return;
#pragma unroll
    for (int k = 1; k < LB; ++k) top = max(top, tops[k][threadIdx.x]);
    atomicMax(wt + b, top);
}
static_assert(LB == 8, "one warp per aux index of a block");

// W's digit slices (layout at t8_at, R = q + ldq l) of RL CN W_l[q, b] over its scale,
// W_l[q, b] = -ck12[b, q] b_pq^l[b, q] + delta_qb tv.
// A thread takes 16 q of one (b, l): 16 loads in flight, coalesced over b, and one
// 16-byte store per slice, contiguous over b; zero digits in the padding
// (q >= nbf5, and R beyond the last aux index: tmp's slices are not written there).
__global__ void __launch_bounds__(256) w_digits_kernel(const double* __restrict__ bpq, const double* __restrict__ ck12,
                                                       const double* __restrict__ tv, int nbf5, int naux, int ldq,
                                                       int nch, const double* __restrict__ RL,
                                                       const double* __restrict__ CN, const double* __restrict__ beta,
                                                       const unsigned* __restrict__ wm,
                                                       const unsigned* __restrict__ wt, int8_t* __restrict__ W8) {
    const int nbp = (nbf5 + 31) / 32 * 32;
    const long long total = (long long)nbp * nch * 8, n55 = (long long)nbf5 * nbf5;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(i / nbp);  // 16 values of R
        const int b = (int)(i - (long long)t * nbp);
        const int l = 16 * t / ldq, q0 = 16 * t - l * ldq;
        if (b >= nbf5) continue;
        const bool in = l < naux;
        const double* B = bpq + n55 * l + b;
        double v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = in && q0 + k < nbf5 ? B[(long long)nbf5 * (q0 + k)] : 0.0;
        const double sc = w_scale(beta[b], wm[b], wt[b]);
        const double f = (sc == 0.0 || !in) ? 0.0 : RL[l] * (F * 0x1p56 / sc);
        const double td = (in && b >= q0 && b < q0 + 16) ? tv[b + (long long)nbf5 * l] : 0.0;
        unsigned wd[4][S];
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
            unsigned long long z[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int q = q0 + 4 * k4 + k;
                double x = 0.0;
                if (q < nbf5) {
                    x = -ck12[b + (long long)nbf5 * q] * v[4 * k4 + k];
                    if (q == b) x += td;
                    x *= CN[q];
                }
                z[k] = digits7(x * f);
            }
            pack4(z, wd[k4]);
        }
        int8_t* dst = W8 + 16 * ((long long)nbf5 * S * t + b);
#pragma unroll
        for (int j = 0; j < S; ++j)
            *reinterpret_cast<uint4*>(dst + 16ll * nbf5 * j) = make_uint4(wd[0][j], wd[1][j], wd[2][j], wd[3][j]);
    }
}

}  // namespace oz

namespace {

int ldn_of(int nbf) { return (nbf + 15) / 16 * 16; }  // 16-byte row pitch (TMA stride rule)
size_t align256(size_t b) { return (b + 255) / 256 * 256; }
// one slice of b (whole 128-row tiles); the job's buffer holds the S slices, sa, RL, RLi
// and the spread of the row norms (two doubles)
size_t slice_bytes(int nbf, int naux) { return ((size_t)naux * nbf + oz::MT - 1) / oz::MT * oz::MT * ldn_of(nbf); }

struct JobLayout {
    size_t sa, rl, spread, bytes;
};
JobLayout job_layout(int nbf, int naux) {
    JobLayout o;
    o.sa = align256(oz::S * slice_bytes(nbf, naux));
    o.rl = o.sa + align256(sizeof(double) * (size_t)nbf * naux);
    o.spread = o.rl + sizeof(double) * 2 * (size_t)naux;
    o.bytes = o.spread + sizeof(double) * 2;
    return o;
}

// C5's slices and the per-column arrays of a call, in job->oz_c
struct CallLayout {
    int nq;
    size_t c2, sb1, sb2, cn, cb, beta, wm, wt, bytes;
};
CallLayout call_layout(int nbf, int nbf5) {
    CallLayout o;
    o.nq = (nbf5 + oz::QT - 1) / oz::QT * oz::QT;
    const size_t col = align256(sizeof(double) * (size_t)o.nq);
    o.c2 = align256((size_t)oz::S * nbf5 * ((nbf + oz::KC - 1) / oz::KC * oz::KC));
    o.sb1 = 2 * o.c2;
    o.sb2 = o.sb1 + col;
    o.cn = o.sb2 + col;
    o.cb = o.cn + col;
    o.beta = o.cb + col;
    o.wm = o.beta + col;
    o.wt = o.wm + sizeof(unsigned) * (size_t)o.nq;
    o.bytes = o.wm + col;
    return o;
}

int ldq_of(int nbf5) { return (nbf5 + 15) / 16 * 16; }
// 128-wide chunks of the (q, l) index
int chunks_of(int nbf5, int naux) { return (int)(((long long)ldq_of(nbf5) * naux + oz::KC - 1) / oz::KC); }

template <int MODE, int NKC>
int launch_one(donof_ctx* ctx, cudaStream_t st, const CUtensorMap& ma, const CUtensorMap& mb, const oz::Params& P,
               int grid) {
    static std::atomic<unsigned long long> attr_mask{0};
    const unsigned long long bit = 1ull << (ctx->device & 63);
    if (!(attr_mask.load(std::memory_order_acquire) & bit)) {
        DONOF_CUDA(ctx, cudaFuncSetAttribute(oz::oz_kernel<MODE, NKC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             oz::SMEM_ALLOC));
        attr_mask.fetch_or(bit, std::memory_order_acq_rel);
    }
    oz::oz_kernel<MODE, NKC><<<grid, oz::NTHREADS, oz::SMEM_ALLOC, st>>>(ma, mb, P); count_launch();
    DONOF_CUDA(ctx, cudaGetLastError());
    return DONOF_OK;
}
// The instance for the call's resident K chunks (0: B streamed).
template <int MODE>
int launch_oz(donof_ctx* ctx, cudaStream_t st, const CUtensorMap& ma, const CUtensorMap& mb, const oz::Params& P,
              int grid) {
    if constexpr (MODE != oz::YSUM) {
        if (P.resident && P.nkc == 1) return launch_one<MODE, 1>(ctx, st, ma, mb, P, grid);
        if (P.resident && P.nkc == 2) return launch_one<MODE, 2>(ctx, st, ma, mb, P, grid);
    }
    return launch_one<MODE, 0>(ctx, st, ma, mb, P, grid);
}

// Parameters common to the products of a call.
oz::Params base_params(donof_job* job, int nbf5) {
    donof_ctx* ctx = job->ctx;
    const JobLayout jl = job_layout(job->nbf, job->naux);
    const CallLayout cl = call_layout(job->nbf, nbf5);
    char* jb = static_cast<char*>(job->oz_b);
    char* cb = job->oz_c.as<char>();
    oz::Params P{};
    P.nbf = job->nbf; P.nbf5 = nbf5; P.naux = job->naux; P.ldq = ldq_of(nbf5);
    P.sa = reinterpret_cast<double*>(jb + jl.sa);
    P.RL = reinterpret_cast<double*>(jb + jl.rl);
    P.RLi = P.RL + job->naux;
    P.sb1 = reinterpret_cast<double*>(cb + cl.sb1);
    P.sb2 = reinterpret_cast<double*>(cb + cl.sb2);
    P.CN = reinterpret_cast<double*>(cb + cl.cn);
    P.cb = reinterpret_cast<double*>(cb + cl.cb);
    P.beta = reinterpret_cast<double*>(cb + cl.beta);
    P.wm = reinterpret_cast<unsigned*>(cb + cl.wm);
    P.wt = reinterpret_cast<unsigned*>(cb + cl.wt);
    P.fail = ctx->fail_dev ? ctx->fail_dev + FAIL_MBAR : nullptr;
    P.wait = sm100::wait_budget(ctx->wait_limit);
    return P;
}

// Tiles, ring and CTAs of a product with K = nbf and C5's slices as B (T1, T2):
// B stays in shared memory where its column tile and at least four A stages fit
// (nbf <= 256) and every column tile has a CTA, else it streams through two stages.
int shape_c5(donof_ctx* ctx, oz::Params& P, long long rows) {
    constexpr int stage = oz::S * oz::BS_BYTES;
    P.nrt = (int)((rows + oz::MT - 1) / oz::MT);
    P.nct = (P.nbf5 + oz::QT - 1) / oz::QT;
    P.nkc = (P.nbf + oz::KC - 1) / oz::KC;
    P.k4_last = (P.nbf - (P.nkc - 1) * oz::KC + 31) / 32;
    const long long units = (long long)P.nrt * P.nct;
    const int grid = (int)(units < ctx_ctas(ctx) ? units : ctx_ctas(ctx));
    P.resident = P.nkc <= 2 && P.nkc * stage + 4 * oz::A_BYTES <= oz::DATA_BYTES && grid >= P.nct;
    P.ring_off = (P.resident ? P.nkc : 2) * stage;
    P.ring = (oz::DATA_BYTES - P.ring_off) / oz::A_BYTES;
    if (P.ring > oz::RING_MAX) P.ring = oz::RING_MAX;
    return grid;
}

// rows x digits of 16-byte groups (C5's slices, W's slices): boxes of 64 rows, every
// digit, the eight groups of a chunk
int map_b(donof_job* job, const void* base, int rows, int chunks, CUtensorMap* m) {
    cuuint64_t dims[3] = {2 * (cuuint64_t)rows, oz::S, 8 * (cuuint64_t)chunks};
    cuuint64_t strides[2] = {16 * (cuuint64_t)rows, 16 * (cuuint64_t)rows * oz::S};
    cuuint32_t box[3] = {2 * oz::QT, oz::S, 8};
    return make_tmap_u64_flat(job->ctx, m, base, 3, dims, strides, box);
}
// C5's truncated (T1) or balanced (T2) slices
int map_c5(donof_job* job, int nbf5, bool balanced, CUtensorMap* m) {
    const char* base = job->oz_c.as<char>() + (balanced ? call_layout(job->nbf, nbf5).c2 : 0);
    return map_b(job, base, nbf5, (job->nbf + oz::KC - 1) / oz::KC, m);
}

// tmp's slices: T2's A operand (MN-major) and Y's (K-major) share the map: boxes of
// 128 m, the eight groups of a chunk of (q, l), one digit
int map_t8(donof_job* job, int nbf5, CUtensorMap* m) {
    const cuuint64_t nbf = job->nbf;
    cuuint64_t dims[3] = {2 * nbf, 8, (cuuint64_t)oz::S * chunks_of(nbf5, job->naux)};
    cuuint64_t strides[2] = {16 * nbf, 128 * nbf};
    cuuint32_t box[3] = {2 * oz::MT, 8, 1};
    return make_tmap_u64_flat(job->ctx, m, job->tmp.ptr, 3, dims, strides, box);
}

// C5's slices and scales (and W's beta where the coefficients are given)
int prep(donof_job* job, cudaStream_t st, const double* C, const double* n, const double* cj12, const double* ck12,
         int nbf5) {
    donof_ctx* ctx = job->ctx;
    const CallLayout cl = call_layout(job->nbf, nbf5);
    DONOF_CHECK(job->oz_c.ensure(ctx, cl.bytes));
    const oz::Params P = base_params(job, nbf5);
    oz::PrepArgs a{};
    a.C = C; a.n = n; a.cj12 = cj12; a.ck12 = ck12;
    a.nbf = job->nbf; a.nbf5 = nbf5; a.nkc = (job->nbf + oz::KC - 1) / oz::KC;
    a.sb1 = const_cast<double*>(P.sb1); a.sb2 = const_cast<double*>(P.sb2);
    a.CN = const_cast<double*>(P.CN); a.cb = const_cast<double*>(P.cb);
    a.beta = const_cast<double*>(P.beta);
    a.c1 = job->oz_c.as<int8_t>(); a.c2 = a.c1 + cl.c2; a.wm = P.wm; a.wt = P.wt;
    oz::prep_kernel<<<cl.nq, 128, 0, st>>>(a); count_launch();
    DONOF_CUDA(ctx, cudaGetLastError());
    return DONOF_OK;
}

// T1 of the call's C5: tmp's digit slices into job->tmp, or tmp in FP64 into `out`.
int t1(donof_job* job, cudaStream_t st, int nbf5, double* out) {
    donof_ctx* ctx = job->ctx;
    const int nbf = job->nbf, naux = job->naux, ldn = ldn_of(nbf);
    CUtensorMap ma, mb;
    {   // b's slices: boxes of 128 rows (m, l), the eight groups of a chunk of n, one digit
        const cuuint64_t groups = ldn / 16, tiles = ((cuuint64_t)nbf * naux + oz::MT - 1) / oz::MT;
        cuuint64_t dims[3] = {2 * oz::MT, groups, tiles * oz::S};
        cuuint64_t strides[2] = {16 * oz::MT, 16 * oz::MT * groups};
        cuuint32_t box[3] = {2 * oz::MT, 8, 1};
        DONOF_CHECK(make_tmap_u64_flat(ctx, &ma, job->oz_b, 3, dims, strides, box));
    }
    DONOF_CHECK(map_c5(job, nbf5, false, &mb));
    oz::Params P = base_params(job, nbf5);
    const int grid = shape_c5(ctx, P, (long long)nbf * naux);
    prof_begin(ctx, st);
    if (out) {
        P.out = out;
        DONOF_CHECK(launch_oz<oz::T1_F64>(ctx, st, ma, mb, P, grid));
    } else {
        P.t8 = job->tmp.as<int8_t>();
        DONOF_CHECK(launch_oz<oz::T1_DIGITS>(ctx, st, ma, mb, P, grid));
    }
    prof_end(ctx, st);
    return DONOF_OK;
}

}  // namespace

// T2 and Y from digits, or as FP64 GEMMs of T1's tmp: those where b's rows differ too much
// in size, and for a few orbitals in a small basis, where the digit route's launches and
// the padding of nbf5 to 64 columns cost more than the products (Lagrangian and JKH_MO in
// us at naux = 4 nbf: nbf = 128, nbf5 = 8 87 and 96 from digits, 69 and 91 as GEMMs; 200
// and 24 152 and 137 against 137 and 127; but 200 and 32 154 and 139 against 152 and 131,
// 200 and 48 174 and 145 against 191 and 146, 256 and 16 173 and 182 against 193 and 184).
bool ozaki_products(const donof_job* job, int nbf5) {
    return job->oz_b && !job->oz_t1_only && (nbf5 > 24 || job->nbf >= 224);
}

bool ozaki_shape_ok(int nbf) { return nbf >= 1 && nbf <= 16384; }

size_t ozaki_bytes(int nbf, int naux) { return job_layout(nbf, naux).bytes; }

// Digit slices and row scales of the job's b (kept until ozaki_free).
int ozaki_build(donof_job* job) {
    donof_ctx* ctx = job->ctx;
    const int nbf = job->nbf, naux = job->naux;
    if (job->oz_b) return DONOF_OK;
    if (!ozaki_shape_ok(nbf)) {
        set_error(ctx, "the tensor-core FP64 transform needs nbf <= 16384 (got %d)", nbf);
        return DONOF_ERR_ARG;
    }
    const JobLayout jl = job_layout(nbf, naux);
    void* buf = nullptr;
    DONOF_CHECK(dev_alloc(ctx, &buf, jl.bytes));
    int8_t* slices = static_cast<int8_t*>(buf);
    double* sa = reinterpret_cast<double*>(static_cast<char*>(buf) + jl.sa);
    double* RL = reinterpret_cast<double*>(static_cast<char*>(buf) + jl.rl);
    double* rn = RL + naux;
    double* rm = static_cast<double*>(buf);  // row norms over l, until the slices take their place
    double *spread = reinterpret_cast<double*>(static_cast<char*>(buf) + jl.spread), norms[2] = {0.0, 0.0};
    cudaStream_t st = ctx->stream;
    cudaError_t e = cudaMemsetAsync(rn, 0, sizeof(double) * (size_t)naux, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(rm, 0, sizeof(double) * (size_t)nbf, st);
    if (e == cudaSuccess) {
        oz::row_scale_kernel<<<8 * ctx->sm_count, 256, 0, st>>>(job->b, nbf, (long long)naux, sa,
                                                               reinterpret_cast<unsigned long long*>(rn),
                                                               reinterpret_cast<unsigned long long*>(rm));
        count_launch();
        oz::row_spread_kernel<<<1, 32, 0, st>>>(rm, nbf, spread); count_launch();
        oz::split_b_kernel<<<16 * ctx->sm_count, 256, 0, st>>>(job->b, sa, nbf, ldn_of(nbf), (long long)naux, slices);
        count_launch();
        oz::row_finish_kernel<<<(naux + 255) / 256, 256, 0, st>>>((long long)naux, RL, rn); count_launch();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(norms, spread, sizeof(norms), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        dev_free(ctx, buf);
        set_error(ctx, "digit slices of b: %s", cudaGetErrorString(e));
        return DONOF_ERR_CUDA;
    }
    job->oz_b = buf;
    job->oz_t1_only = norms[0] > oz::ROW_SPREAD * norms[1];
    ++job->oz_gen;
    return DONOF_OK;
}

void ozaki_free(donof_job* job) {
    if (!job->oz_b) return;
    cudaStreamSynchronize(job->ctx->stream);
    dev_free(job->ctx, job->oz_b);
    job->oz_b = nullptr;
    job->oz_c.release(job->ctx);
    ++job->oz_gen;
}

// tmp_l = B_l C5 for every l (FP64 result, tmp[m + nbf*q + nbf*nbf5*l]).
int t1_ozaki(donof_job* job, cudaStream_t st, const double* C, int nbf5, double* tmp) {
    DONOF_CHECK(prep(job, st, C, nullptr, nullptr, nullptr, nbf5));
    return t1(job, st, nbf5, tmp);
}

// T1 and T2: tmp's digit slices into job->tmp, b_pq into job->bpq.  n, cj12 and
// ck12 (or null) are the coefficients of the W that y_ozaki will build.
int transforms_ozaki(donof_job* job, cudaStream_t st, const double* C, const double* n, const double* cj12,
                     const double* ck12, int nbf5) {
    donof_ctx* ctx = job->ctx;
    const int nbf = job->nbf, naux = job->naux;
    DONOF_CHECK(job->tmp.ensure(ctx, (size_t)oz::S * nbf * oz::KC * chunks_of(nbf5, naux)));
    // b_pq, and its diagonals again behind it
    DONOF_CHECK(job->bpq.ensure(ctx, sizeof(double) * (size_t)nbf5 * (nbf5 + 1) * naux));
    DONOF_CHECK(prep(job, st, C, n, cj12, ck12, nbf5));
    DONOF_CHECK(t1(job, st, nbf5, nullptr));
    CUtensorMap ma, mb;
    DONOF_CHECK(map_t8(job, nbf5, &ma));
    DONOF_CHECK(map_c5(job, nbf5, true, &mb));
    oz::Params P = base_params(job, nbf5);
    const int grid = shape_c5(ctx, P, (long long)P.ldq * naux);
    P.out = job->bpq.as<double>();
    P.diag = P.out + (size_t)nbf5 * nbf5 * naux;
    if (n == nullptr) P.wm = nullptr;
    return launch_oz<oz::T2>(ctx, st, ma, mb, P, grid);
}

// W from job->bpq and Y = sum_l tmp_l W_l as FP64 partials (nbf x nbf5 each) in
// job->part, after transforms_ozaki with the same coefficients.
int y_ozaki(donof_job* job, cudaStream_t st, const double* n, const double* cj12, const double* ck12, int nbf5,
            int nalpha, int nbeta, const double** ypart, int* nparts, unsigned* tail_words) {
    donof_ctx* ctx = job->ctx;
    const int nbf = job->nbf, naux = job->naux, ldq = ldq_of(nbf5), nch = chunks_of(nbf5, naux);
    const size_t wbytes = (size_t)oz::S * nbf5 * oz::KC * nch;
    const size_t o_tv = align256(wbytes);
    DONOF_CHECK(job->W.ensure(ctx, o_tv + sizeof(double) * (size_t)nbf5 * naux));
    int8_t* w8 = job->W.as<int8_t>();
    double* tv = reinterpret_cast<double*>(job->W.as<char>() + o_tv);
    oz::Params P = base_params(job, nbf5);
    const double* bpq = job->bpq.as<double>();
    {
        const dim3 grid((naux + oz::LB - 1) / oz::LB, (nbf5 + 31) / 32);
        oz::diag_kernel<<<grid, 256, 0, st>>>(bpq + (size_t)nbf5 * nbf5 * naux, n, cj12, nbf5, naux, nalpha, nbeta,
                                              P.RL, P.CN, tv, P.wt, tail_words);
        count_launch();
    }
    {
        const long long items = (long long)((nbf5 + 31) / 32 * 32) * nch * 8;
        long long blocks = (items + 255) / 256;
        if (blocks > 16LL * ctx->sm_count) blocks = 16LL * ctx->sm_count;
        oz::w_digits_kernel<<<(int)blocks, 256, 0, st>>>(bpq, ck12, tv, nbf5, naux, ldq, nch, P.RL, P.CN, P.beta, P.wm,
                                                       P.wt, w8);
        count_launch();
    }
    DONOF_CUDA(ctx, cudaGetLastError());

    constexpr int stage = oz::S * oz::BS_BYTES;
    P.nrt = (nbf + oz::MT - 1) / oz::MT;
    P.nct = (nbf5 + oz::QT - 1) / oz::QT;
    P.nkc = nch;
    P.k4_last = (int)(((long long)ldq * naux - (long long)(nch - 1) * oz::KC + 31) / 32);
    P.ring_off = 2 * stage;
    P.ring = (oz::DATA_BYTES - P.ring_off) / oz::A_BYTES;
    if (P.ring > oz::RING_MAX) P.ring = oz::RING_MAX;
    // The split of K: waves of units over the SMs, each unit a few chunks (about 3.5
    // us each, and 2 us to fill and drain), and the partials written and summed by
    // the tail.  A rule of the shape alone, so that a shape sums in one order.
    const int tiles = P.nrt * P.nct;
    double best = 0.0;
    for (int s = 1; s <= P.nkc && s <= 1024; ++s) {
        const int cpu = (P.nkc + s - 1) / s;
        if (cpu > oz::KMAX_CHUNKS) continue;
        const int used = (P.nkc + cpu - 1) / cpu;
        const long long waves = ((long long)tiles * used + ctx->sm_count - 1) / ctx->sm_count;
        const double cost = waves * (3.5 * cpu + 2.0) + used * ((double)nbf * nbf5 * 16.0 / 3e6);
        if (best == 0.0 || cost < best) {
            best = cost;
            P.cpu = cpu;
            P.nsplit = used;
        }
    }
    if (best == 0.0) {  // more than 1024 units of the longest exact range
        P.cpu = oz::KMAX_CHUNKS;
        P.nsplit = (P.nkc + P.cpu - 1) / P.cpu;
    }
    DONOF_CHECK(job->part.ensure(ctx, sizeof(double) * (size_t)P.nsplit * nbf * nbf5));
    P.out = job->part.as<double>();
    CUtensorMap ma, mb;
    DONOF_CHECK(map_t8(job, nbf5, &ma));
    DONOF_CHECK(map_b(job, w8, nbf5, nch, &mb));
    const long long units = (long long)tiles * P.nsplit;
    const int grid = (int)(units < ctx_ctas(ctx) ? units : ctx_ctas(ctx));
    DONOF_CHECK(launch_oz<oz::YSUM>(ctx, st, ma, mb, P, grid));
    *ypart = job->part.as<double>();
    *nparts = P.nsplit;
    return DONOF_OK;
}

}  // namespace donof
