// Symmetric eigen-decomposition on the device for Iaux (src/integrals.jl:68-91,
// ext/DoNOFGPUExt.jl:9-33: eigen(Symmetric(G))) by the parallel cyclic
// Jacobi method in blocks: two-sided plane rotations on disjoint index pairs, the
// rotation angle by Rutishauser's formulas (t = sign(theta) / (|theta| +
// sqrt(1 + theta^2)), theta = (a_qq - a_pp) / (2 a_pq)), and a pair skipped when
// |a_pq| <= eps sqrt(|a_pp a_qq|) (the relative test of Demmel and Veselic).
//
// The indices (padded with zeros to a multiple of 64) are cut into blocks of 32.  A
// round pairs the blocks by the round-robin (circle) ordering of Brent and Luk
// (J. Sci. Stat. Comput. 6, 1985).  One cooperative kernel runs every sweep; a round
// has two phases between bounded grid barriers (dtile.cuh):
//   A  a CTA per block pair rotates the pair's 64 x 64 diagonal block in shared
//      memory, accumulating the rotations in a 64 x 64 Q: in a sweep's first round
//      all 63 x 32 index pairs (circle ordering; those of a smaller matrix alone: Iaux
//      at naux = 8 495 us with all of them, 224 so), in the others the 32 x 32 pairs
//      across the two blocks (32 steps of 32 disjoint pairs).  A sweep visits
//      every index pair outside the blocks once, and those inside once.
//   B  the other 64 x 64 blocks of A become Q1^T A_blk Q2 and V's column pairs V Q,
//      one tile per CTA step on the FP64 tensor cores (m16n8k4); tiles whose pairs
//      rotated nothing are skipped.
// The iteration stops after the first sweep that rotates no pair; a sweep count
// above the limit is reported as non-convergence.  A well-conditioned G takes 10 to 16
// sweeps.  Where eigenvalues lie below the rounding of G, the noise that the products of
// phase B leave beside them is rotated away over many more: 41 to 55 for eigenvalues over
// 16 to 20 decades, or functions that stand in a badly scaled set twice, at n = 512 to 3008
// (single rotations ended some of these within 40).
//
// What bounds it: the chain of rotation steps, 511 a sweep and 16 sweeps at n = 512,
// about 0.8 us each (the angle 460 cycles, the 2 x 2 blocks 960, most of it shared-
// memory traffic).  Measured on one B200: n = 512 9.9 ms (67 ms with single rotations
// over the whole matrix, where a step was a grid-wide round: two grid barriers and
// strided 2 x 2 blocks in L2), Iaux at naux = 1024 32 ms (334), 2048 125 ms (1977).
#include <math.h>

#include <atomic>

#include "dtile.cuh"
#include "kernels.cuh"

namespace donof {

namespace {

constexpr int EIG_THREADS = 384;    // eight warps on A (or on a tile's product), four on Q
constexpr int SW_THREADS = 256;
constexpr int EIG_MAX_SWEEPS = 128;  // see the end of the comment above
constexpr double EIG_EPS = 2.220446049250313e-16;
constexpr int EB = 32;            // block
constexpr int PB = 2 * EB;        // block pair
constexpr int NBLK2 = EB * (EB - 1) / 2;  // 2 x 2 blocks of a step below the diagonal ones, two a thread
constexpr int LD = PB + 4;        // shared-memory leading dimension (4 mod 16 doubles: conflict-free fragments)
constexpr int LDS = PB + 1;       // ... of the block being rotated (its rows and its columns are read across lanes)
constexpr int EIG_SMEM = 3 * PB * LD * (int)sizeof(double);
static_assert(NBLK2 <= 2 * SW_THREADS && EIG_THREADS == SW_THREADS + 2 * PB, "roles");

struct EigState {
    dtile::GridSync gs;
    int rotations[EIG_MAX_SWEEPS];  // per sweep, zeroed before the launch
    int sweeps;                     // sweeps run, the last one without a rotation
    int converged;
};

struct EigArgs {
    double* A;      // N x N, symmetric (both triangles), overwritten: diagonal = eigenvalues
    double* V;      // N x N eigenvectors (columns), starts as the identity
    double* Q;      // P matrices of 64 x 64 (column-major), the round's rotations
    int* rotated;   // P flags of the round
    EigState* st;
    int n, N, P;    // size, padded size, block pairs
    dtile::WaitCtl wc;
};

// Index at position pos of round r < n - 1 of the circle ordering of n (position 0 fixed).
__device__ __forceinline__ int circle(int pos, int r, int n) {
    const int x = pos + r;
    return pos == 0 ? 0 : x < n ? x : x - (n - 1);
}

// Blocks I < J of pair p in round r.
__device__ __forceinline__ void block_pair(int p, int r, int nb, int& I, int& J) {
    const int a = circle(p, r, nb), b = circle(nb - 1 - p, r, nb);
    I = a < b ? a : b;
    J = a < b ? b : a;
}
// Global index of local index x (0..63) of the pair (I, J).
__device__ __forceinline__ int global_index(int x, int I, int J) { return x < EB ? I * EB + x : J * EB + x - EB; }

// |a_pq| > eps sqrt(|a_pp a_qq|), squared (the square root would head the step's
// chain of dependent operations).
__device__ __forceinline__ bool needs_rotation(double app, double aqq, double apq) {
    const double m = fabs(app * aqq);
    return m > 0.0 ? apq * apq > EIG_EPS * EIG_EPS * m : apq != 0.0;
}

// Rotation (c, s) of theta = d / e with t = sign(theta) / (|theta| + sqrt(1 + theta^2))
// = +-e / (|d| + sqrt(d^2 + e^2)).  The angle needs few digits (it only decides how far
// a_pq falls: here by 1e-7, and every element of the pair's block is formed with the
// c and s that are used), so t is formed in FP32 and then taken as exact; c = 1/sqrt(1
// + t^2) and s = t c carry FP64, so the rotation is orthogonal to FP64 rounding.  In
// FP64 throughout the angle took 630 cycles of a step, so 460; the sweeps stay the same.
__device__ __forceinline__ double2 rotation(double d, double e) {
    const int hi = max(__double2hiint(d) & 0x7ff00000, __double2hiint(e) & 0x7ff00000);
    const double f = __hiloint2double(max(0x7fd00000 - hi, 0x00100000), 0);  // the larger one to [1/2, 1), exactly
    d *= f;
    e *= f;
    const float df = fabsf((float)d), ef = fabsf((float)e);
    const float tf = __fdividef(ef, df + sqrtf(fmaf(df, df, ef * ef)));
    double t = (double)tf;
    float y0 = rsqrtf(fmaf(tf, tf, 1.0f));
    if (tf < 1e-18f) t = 0.5 * fabs(e) / fabs(d);  // below what FP32 resolves: t = e / (2 d)
    // 1/sqrt(x) from the FP32 value: y (1 + h/2 + 3 h^2/8), h = 1 - x y^2 ~ 1e-7
    const double y = (double)y0, h = fma(-fma(t, t, 1.0), y * y, 1.0);
    const double c = fma(fma(h, 0.375, 0.5), h * y, y);
    return make_double2(c, (d >= 0.0) == (e >= 0.0) ? t * c : -t * c);
}

// Barriers of the whole block for warps in different branches (__syncthreads is defined
// only where every warp takes the same branch): named barrier 1, counted by threads, in
// whole warps.  role_any also tells whether a thread passed true.
__device__ __forceinline__ void role_sync() { asm volatile("barrier.cta.sync.aligned 1, %0;" ::"n"(EIG_THREADS) : "memory"); }
__device__ __forceinline__ bool role_any(bool x) {
    int any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.s32 p, %1, 0;\n\t"
        "barrier.cta.red.or.pred.aligned q, 1, %2, p;\n\t"
        "selp.s32 %0, 1, 0, q;\n\t}"
        : "=r"(any)
        : "r"((int)x), "n"(EIG_THREADS)
        : "memory");
    return any != 0;
}

// Phase A for one pair: rotates its diagonal block of A, writes the block and Q.
// sm: S (lower triangle, [max][min]) and Q ([column][row]).  Warp 0 forms a step's
// rotations; warps 0-7 apply them to S; warps 8-11 to Q, two neighbouring lanes per
// row: in the steps across the blocks the row lives in their registers (16 columns of
// either block each), the second block's columns shifted by one a step, with one
// exchange between the two lanes, so that rotation j always meets register j.
__device__ void rotate_pair(const EigArgs& a, int p, int r, int sweep, double* sm) {
    __shared__ double2 rcs[EB];  // c, s of the step's rotations ((1, 0): none)
    __shared__ int rpq[EB];      // p | q << 8
    double* S = sm;
    double* Q = sm + PB * LD;
    const int tid = threadIdx.x;
    int I, J;
    block_pair(p, r, 2 * a.P, I, J);
    auto at = [&](int x, int y) -> double& { return x > y ? S[x * LDS + y] : S[y * LDS + x]; };
    for (int e = tid; e < PB * PB; e += EIG_THREADS) {
        const int x = e & (PB - 1), y = e / PB;
        if (x >= y) S[x * LDS + y] = a.A[global_index(x, I, J) + (long long)a.N * global_index(y, I, J)];
        if (r == 0) Q[y * LD + x] = x == y ? 1.0 : 0.0;
    }
    int count = 0;  // thread < 32: rotations made
    __syncthreads();
    // a step's rotation of pair (x, y) of this lane, and its 2 x 2 diagonal block
    // behind it (elements of no other 2 x 2 block of the step)
    double app, aqq, apq;
    double2 cs;
    int lo, hi;
    auto form = [&](int x, int y) {
        lo = min(x, y);
        hi = max(x, y);
        app = S[lo * LDS + lo];
        aqq = S[hi * LDS + hi];
        apq = S[hi * LDS + lo];
        const bool act = needs_rotation(app, aqq, apq);
        cs = rotation(aqq - app, 2.0 * apq);
        if (!act) cs = make_double2(1.0, 0.0);
        rcs[tid] = cs;
        rpq[tid] = lo | hi << 8;
        count += act;
        return (int)act;
    };
    auto keep = [&]() {
        const double c = cs.x, s = cs.y;
        const double m0 = c * app - s * apq, m1 = s * app + c * apq, m2 = c * apq - s * aqq, m3 = s * apq + c * aqq;
        S[lo * LDS + lo] = c * m0 - s * m2;
        S[hi * LDS + lo] = c * m1 - s * m3;
        S[hi * LDS + hi] = s * m1 + c * m3;
    };
    // this thread's 2 x 2 blocks: rotations k1 > k2
    int k1[2], k2[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        k1[u] = 1;
        k2[u] = tid + u * (NBLK2 / 2);
        while (k2[u] >= k1[u]) k2[u] -= k1[u]++;
    }
    auto apply = [&]() {
        if (tid >= NBLK2 / 2) return;
        double *e[2][4], x[2][4];
        double2 r1[2], r2[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {  // every load before the stores
            // rows {p1, q1} of rotation k2, columns {p2, q2} of rotation k1
            const int w1 = rpq[k2[u]], w2 = rpq[k1[u]];
            const int p1 = w1 & 255, q1 = w1 >> 8, p2 = w2 & 255, q2 = w2 >> 8;
            r1[u] = rcs[k2[u]];
            r2[u] = rcs[k1[u]];
            e[u][0] = &at(p1, p2);
            e[u][1] = &at(p1, q2);
            e[u][2] = &at(q1, p2);
            e[u][3] = &at(q1, q2);
#pragma unroll
            for (int v = 0; v < 4; ++v) x[u][v] = *e[u][v];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            // M = X J2, then J1^T M  (J = [[c, s], [-s, c]] on {p, q})
            const double m00 = x[u][0] * r2[u].x - x[u][1] * r2[u].y, m01 = x[u][0] * r2[u].y + x[u][1] * r2[u].x;
            const double m10 = x[u][2] * r2[u].x - x[u][3] * r2[u].y, m11 = x[u][2] * r2[u].y + x[u][3] * r2[u].x;
            *e[u][0] = r1[u].x * m00 - r1[u].y * m10;
            *e[u][1] = r1[u].x * m01 - r1[u].y * m11;
            *e[u][2] = r1[u].y * m00 + r1[u].x * m10;
            *e[u][3] = r1[u].y * m01 + r1[u].x * m11;
        }
    };
    if (r == 0) {
        const int i = (tid - SW_THREADS) >> 1, j0 = EB / 2 * (tid & 1);  // row of Q, first rotation
        double* row = Q + i;
        // (a matrix smaller than the block: the circle of its own indices, the others idle)
        const int ring = a.P == 1 ? (a.n + 1) & ~1 : PB;
        if (tid < EB && tid >= ring / 2) {
            rcs[tid] = make_double2(1.0, 0.0);
            rpq[tid] = 2 * tid | (2 * tid + 1) << 8;
        }
        for (int k = 0; k < ring - 1; ++k) {
            int act = 0;
            if (tid < ring / 2) act = form(circle(tid, k, ring), circle(ring - 1 - tid, k, ring));
            if (!__syncthreads_or(act)) continue;
            if (tid < SW_THREADS) {
                if (tid < ring / 2) keep();
                apply();
            } else {
                constexpr int U = 8;  // loads of U rotations before their stores
                for (int j = j0; j < j0 + EB / 2; j += U) {
                    double *x[U], *y[U], vx[U], vy[U];
                    double2 cs[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int pq = rpq[j + u];
                        cs[u] = rcs[j + u];
                        x[u] = row + (pq & 255) * LD;
                        y[u] = row + (pq >> 8) * LD;
                        vx[u] = *x[u];
                        vy[u] = *y[u];
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        *x[u] = cs[u].x * vx[u] - cs[u].y * vy[u];
                        *y[u] = cs[u].y * vx[u] + cs[u].x * vy[u];
                    }
                }
            }
            __syncthreads();
        }
    } else if (tid < SW_THREADS) {  // (one loop for both roles, under block barriers: 5% slower)
        for (int k = 0; k < EB; ++k) {
            int act = 0;
            if (tid < EB) act = form(tid, EB + ((tid + k) & (EB - 1)));
            const bool any = role_any(act);
            if (any) {
                if (tid < EB) keep();
                apply();
            }
            role_sync();
        }
    } else {
        constexpr int H = EB / 2;
        const int i = (tid - SW_THREADS) >> 1, j0 = H * (tid & 1);  // row of Q, first rotation
        double x[H], y[H];  // columns j0 + j, and EB + (j0 + j + k) % EB
#pragma unroll
        for (int j = 0; j < H; ++j) {
            x[j] = i == j0 + j ? 1.0 : 0.0;
            y[j] = i == EB + j0 + j ? 1.0 : 0.0;
        }
        for (int k = 0; k < EB; ++k) {
            if (role_any(false)) {
#pragma unroll
                for (int j = 0; j < H; ++j) {
                    const double2 cs = rcs[j0 + j];
                    const double vx = x[j], vy = y[j];
                    x[j] = cs.x * vx - cs.y * vy;
                    y[j] = cs.y * vx + cs.x * vy;
                }
            }
            const double first = __shfl_xor_sync(0xffffffffu, y[0], 1);
#pragma unroll
            for (int j = 0; j < H - 1; ++j) y[j] = y[j + 1];
            y[H - 1] = first;
            role_sync();
        }
#pragma unroll
        for (int j = 0; j < H; ++j) {  // after EB steps y is in place
            Q[(j0 + j) * LD + i] = x[j];
            Q[(EB + j0 + j) * LD + i] = y[j];
        }
    }
    if (tid < EB) {
        for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
        if (tid == 0) {
            a.rotated[p] = count;
            if (count) atomicAdd(&a.st->rotations[sweep], count);
        }
    }
    __syncthreads();
    for (int e = tid; e < PB * PB; e += EIG_THREADS) {
        const int x = e & (PB - 1), y = e / PB;
        a.A[global_index(x, I, J) + (long long)a.N * global_index(y, I, J)] = at(x, y);
        a.Q[(long long)p * PB * PB + e] = Q[y * LD + x];
    }
    __syncthreads();
}

// 64 x 64 x 64 product of shared-memory operands: warp w of the first eight the 16 x 32
// tile (w % 4, w / 4); A(i, k) = A[i sa_i + k sa_k], B(k, j) = B[j LD + k].
constexpr int PN = 4;  // n8 blocks of a warp's tile
__device__ __forceinline__ void product(const double* A, int sa_i, int sa_k, const double* B, double (&acc)[PN][4]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int i0 = 16 * (w & 3), j0 = 8 * PN * (w >> 2);
    if (w >= 8) return;
#pragma unroll
    for (int n = 0; n < PN; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = 0.0;
#pragma unroll 4
    for (int k = 0; k < PB; k += 4) {
        const double a0 = A[(i0 + g) * sa_i + (k + t) * sa_k], a1 = A[(i0 + g + 8) * sa_i + (k + t) * sa_k];
#pragma unroll
        for (int n = 0; n < PN; ++n) gemm_detail::mma_f64_16x8x4(acc[n], a0, a1, B[(j0 + 8 * n + g) * LD + k + t]);
    }
}

// Phase B, tile t: pair tiles p2 < p1 of A first, then 64-row chunks of V's column pairs.
__device__ void update_tile(const EigArgs& a, int t, int r, double* sm) {
    double *X = sm, *Q1 = sm + PB * LD, *Q2 = sm + 2 * PB * LD;
    const int tid = threadIdx.x, nt = a.P * (a.P - 1) / 2;
    const int lane = tid & 31, w = tid >> 5, g = lane >> 2, tq = lane & 3;
    const int i0 = 16 * (w & 3), j0 = 8 * PN * (w >> 2);
    const long long N = a.N;
    const bool mine = w < 8;  // this warp holds a part of the products
    double acc[PN][4];
    if (t < nt) {
        int p1 = 1, p2 = t;
        while (p2 >= p1) p2 -= p1++;
        if (!a.rotated[p1] && !a.rotated[p2]) return;  // (the same in every thread)
        int I1, J1, I2, J2;  // rows: pair p2, columns: pair p1
        block_pair(p2, r, 2 * a.P, I1, J1);
        block_pair(p1, r, 2 * a.P, I2, J2);
        const double* q1 = a.Q + (long long)p2 * PB * PB;
        const double* q2 = a.Q + (long long)p1 * PB * PB;
        for (int e = tid; e < PB * PB; e += EIG_THREADS) {
            const int x = e & (PB - 1), y = e / PB;
            X[y * LD + x] = a.A[global_index(x, I1, J1) + N * global_index(y, I2, J2)];
            Q1[y * LD + x] = q1[e];
            Q2[y * LD + x] = q2[e];
        }
        __syncthreads();
        product(Q1, LD, 1, X, acc);  // T(i, j) = sum_k Q1(k, i) X(k, j)
        __syncthreads();
        if (mine) {
#pragma unroll
            for (int n = 0; n < PN; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)  // T as [i][k]
                    X[(i0 + g + 8 * (e >> 1)) * LD + j0 + 8 * n + 2 * tq + (e & 1)] = acc[n][e];
        }
        __syncthreads();
        product(X, LD, 1, Q2, acc);
        if (mine) {
#pragma unroll
            for (int n = 0; n < PN; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int gi = global_index(i0 + g + 8 * (e >> 1), I1, J1);
                    const int gj = global_index(j0 + 8 * n + 2 * tq + (e & 1), I2, J2);
                    a.A[gi + N * gj] = acc[n][e];
                    a.A[gj + N * gi] = acc[n][e];
                }
        }
    } else {
        const int v = t - nt, p = v % a.P, row0 = v / a.P * PB;
        if (!a.rotated[p]) return;
        int I, J;
        block_pair(p, r, 2 * a.P, I, J);
        const double* q = a.Q + (long long)p * PB * PB;
        for (int e = tid; e < PB * PB; e += EIG_THREADS) {
            const int x = e & (PB - 1), y = e / PB;
            X[y * LD + x] = a.V[row0 + x + N * global_index(y, I, J)];  // X(i, k) at [k][i]
            Q1[y * LD + x] = q[e];
        }
        __syncthreads();
        product(X, 1, LD, Q1, acc);
        if (mine) {
#pragma unroll
            for (int n = 0; n < PN; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    a.V[row0 + i0 + g + 8 * (e >> 1) + N * global_index(j0 + 8 * n + 2 * tq + (e & 1), I, J)] = acc[n][e];
        }
    }
    __syncthreads();  // the buffers are free
}

__global__ void __launch_bounds__(EIG_THREADS, 1) jacobi_kernel(const EigArgs a) {
    extern __shared__ __align__(16) double sm[];
    unsigned epoch = 0;
    const unsigned members = gridDim.x;
    const int nb = 2 * a.P, rounds = nb - 1;
    const int tiles = a.P * (a.P - 1) / 2 + a.P * (a.N / PB);
    int sweep = 0;
    bool ok = true, done = false;
    for (; sweep < EIG_MAX_SWEEPS && ok && !done; ++sweep) {
        for (int r = 0; r < rounds && ok; ++r) {
            for (int p = blockIdx.x; p < a.P; p += gridDim.x) rotate_pair(a, p, r, sweep, sm);
            if (!dtile::grid_barrier(&a.st->gs, epoch, members, a.wc)) { ok = false; break; }
            for (int t = blockIdx.x; t < tiles; t += gridDim.x) update_tile(a, t, r, sm);
            if (!dtile::grid_barrier(&a.st->gs, epoch, members, a.wc)) { ok = false; break; }
        }
        if (ok) done = *(volatile int*)&a.st->rotations[sweep] == 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.st->sweeps = sweep;
        a.st->converged = (ok && done) ? 1 : 0;
    }
}

// A = Symmetric(G) (upper triangle of the column-major n x n G) padded with zeros to
// N x N, V = identity.
__global__ void eig_init_kernel(const double* __restrict__ G, int n, int N, double* __restrict__ A,
                                double* __restrict__ V) {
    const long long total = (long long)N * N;
    for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(idx % N), j = (int)(idx / N);
        A[idx] = (i < n && j < n) ? G[min(i, j) + (long long)n * max(i, j)] : 0.0;
        V[idx] = (i == j) ? 1.0 : 0.0;
    }
}

__global__ void eig_diag_kernel(const double* __restrict__ A, int n, int N, double* __restrict__ w) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        w[i] = A[i + (long long)N * i];
}

size_t align256(size_t b) { return (b + 255) / 256 * 256; }

}  // namespace

int eigh_padded(int n) { return (n + PB - 1) / PB * PB; }

size_t eigh_scratch_bytes(int n) {
    const size_t P = eigh_padded(n) / PB;
    return align256(sizeof(EigState)) + align256(sizeof(double) * P * PB * PB) + align256(sizeof(int) * P);
}

// Enqueues the decomposition of Symmetric(G): eigenvalues w (unsorted) and
// eigenvectors V (columns; A and V hold N x N, N = eigh_padded(n), leading dimension
// N); `scratch` eigh_scratch_bytes(n) of device memory.  eigh_finish, after it,
// synchronises and reports.
int eigh_jacobi(donof_ctx* ctx, cudaStream_t st, const double* G, int n, double* A, double* V, double* w,
                void* scratch) {
    const int N = eigh_padded(n), P = N / PB;
    char* base = static_cast<char*>(scratch);
    EigState* es = reinterpret_cast<EigState*>(base);
    double* Q = reinterpret_cast<double*>(base + align256(sizeof(EigState)));
    int* rotated = reinterpret_cast<int*>(base + align256(sizeof(EigState)) + align256(sizeof(double) * (size_t)P * PB * PB));
    long long blocks = ((long long)N * N + 255) / 256;
    if (blocks > 8LL * ctx->sm_count) blocks = 8LL * ctx->sm_count;
    eig_init_kernel<<<(int)blocks, 256, 0, st>>>(G, n, N, A, V); count_launch();
    DONOF_CUDA(ctx, cudaGetLastError());
    DONOF_CUDA(ctx, cudaMemsetAsync(es, 0, sizeof(EigState), st));
    static std::atomic<unsigned long long> attr_mask{0};
    const unsigned long long bit = 1ull << (ctx->device & 63);
    if (!(attr_mask.load(std::memory_order_acquire) & bit)) {
        DONOF_CUDA(ctx, cudaFuncSetAttribute(jacobi_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, EIG_SMEM));
        attr_mask.fetch_or(bit, std::memory_order_acq_rel);
    }
    int per_sm = 0;
    DONOF_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, jacobi_kernel, EIG_THREADS, EIG_SMEM));
    if (per_sm < 1) {
        set_error(ctx, "jacobi_kernel does not fit on an SM");
        return DONOF_ERR_CUDA;
    }
    const int tiles = P * (P - 1) / 2 + P * (N / PB);
    int grid = ctx_ctas(ctx);  // at most one CTA per SM: co-resident (the kernel has grid barriers)
    if (grid > tiles) grid = tiles;
    EigArgs a{A, V, Q, rotated, es, n, N, P, dtile::wait_ctl(ctx)};
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(EIG_THREADS);
    cfg.dynamicSmemBytes = EIG_SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    DONOF_CUDA(ctx, cudaLaunchKernelEx(&cfg, jacobi_kernel, a));
    count_launch();
    eig_diag_kernel<<<(n + 255) / 256, 256, 0, st>>>(A, n, N, w); count_launch();
    DONOF_CUDA(ctx, cudaGetLastError());
    return DONOF_OK;
}

// Synchronises the stream; DONOF_ERR_STATE if the sweeps of the decomposition that
// used `scratch` did not converge, DONOF_ERR_TIMEOUT if a grid barrier ran out.
int eigh_finish(donof_ctx* ctx, cudaStream_t st, const void* scratch) {
    const EigState* es = static_cast<const EigState*>(scratch);
    int hs[2] = {0, 0};
    DONOF_CUDA(ctx, cudaMemcpyAsync(hs, &es->sweeps, sizeof(hs), cudaMemcpyDeviceToHost, st));
    DONOF_CHECK(sync_and_check(ctx));
    if (!hs[1]) {
        set_error(ctx, "Jacobi eigen-decomposition of G did not converge in %d sweeps", hs[0]);
        return DONOF_ERR_STATE;
    }
    return DONOF_OK;
}

}  // namespace donof
