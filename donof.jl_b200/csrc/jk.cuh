// Partial sums of J_MO and K_MO (src/integrals.jl:161-166) over a chunk of aux
// indices from b_pq in FP64 or FP32, accumulated in FP64:
//   part[c][0][p + nbf5 q] = sum_l d_p^l d_q^l,  part[c][1][p + nbf5 q] = sum_l (b_pq^l)^2
// with d_q^l = b_qq^l.  A thread takes JE (p, q) and sums its chunk's l in order.
// Bound by reading b_pq.  The diagonals of JL aux indices at a time are staged in
// shared memory, for nbf5 up to JD; a diagonal element is a 32-byte sector of its own,
// and with one (p, q) per thread the blocks of a chunk fetched it nbf5^2 / 256 times
// (142 us at nbf5 = 160, naux = 928 for 190 MB; 62 us with JE = 4, 157 before staging).
#pragma once

#include "kernels.cuh"

namespace donof {
namespace jk {

constexpr int JT = 256;          // threads
constexpr int JL = 8;            // aux indices staged
constexpr int JV = 4;            // ... and their b_pq loads in flight per (p, q)
constexpr int JD = 512;          // largest nbf5 staged (32 KB)

// (p, q) per thread: four with staged diagonals, or one with direct loads where there
// are few blocks along (p, q) (four a thread would need more chunks of l, whose
// partials a second kernel sums in order: JKH_MO at nbf5 = 60 62 us, 64 with staging)
// and where the diagonals are long (the kernel alone, four against one: FP32 at nbf5 =
// 300, naux = 400 172 and 203 us, at 360 245 and 207, at 400 330 and 211; FP64 at 400
// 240 and 212, at 450, naux = 200 146 and 215, at 512 226 and 214; beyond JD four with
// direct loads took 304 and 137 us at 600, 200 and 100, in the two types, one 304 and 125).
template <class T>
int per_thread(int nbf5) {
    return nbf5 <= (sizeof(T) == 4 ? 320 : JD) && (long long)nbf5 * nbf5 >= 8192 ? 4 : 1;
}
// blocks along (p, q); chunk of l for two or three blocks per SM
template <class T>
int blocks(int nbf5) {
    const long long span = (long long)per_thread<T>(nbf5) * JT;
    return (int)(((long long)nbf5 * nbf5 + span - 1) / span);
}
template <class T>
int chunk(int nbf5, int naux, int sms) {
    const int want = (per_thread<T>(nbf5) == 4 ? 3 : 2) * sms;
    int n = (want + blocks<T>(nbf5) - 1) / blocks<T>(nbf5);
    if (n > naux) n = naux;
    if (n < 1) n = 1;
    return (naux + n - 1) / n;
}

// Stages the diagonals of nl aux indices (B: the first one's b_pq, n of np elements
// from element p0 on) as sd[k ks + q qs]; U loads of a thread in flight together, since
// each is a sector of its own from wherever b_pq lies (one at a time, a group of eight
// aux indices cost eight memory latencies).
template <int U, class T, class S>
__device__ __forceinline__ void stage_diagonals(const T* __restrict__ B, int nbf5, int p0, int np, int nl, S* sd, int ks,
                                                int qs) {
    const long long n55 = (long long)nbf5 * nbf5;
    const int total = nl * np;
    for (int i0 = threadIdx.x; i0 < total; i0 += U * blockDim.x) {
        T r[U];
        int at[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * blockDim.x, k = i / np, q = i - k * np;
            at[u] = i < total ? k * ks + q * qs : -1;
            r[u] = i < total ? B[n55 * k + (long long)(p0 + q) * (nbf5 + 1)] : T(0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (at[u] >= 0) sd[at[u]] = (S)r[u];
    }
}

template <class T, int JE>
__global__ void __launch_bounds__(JT) partial_kernel(const T* __restrict__ bpq, int nbf5, int naux, int lchunk,
                                                     double* __restrict__ part) {
    __shared__ double sd[JE == 1 ? 1 : JL][JE == 1 ? 1 : JD];  // (32 KB would cost direct loads a block per SM)
    const long long n55 = (long long)nbf5 * nbf5, base = blockIdx.x * (long long)(JE * JT) + threadIdx.x;
    const int c = blockIdx.y;
    const int l0 = c * lchunk, l1 = min(naux, l0 + lchunk);
    int p[JE], q[JE];
    double sj[JE], sk[JE];
#pragma unroll
    for (int j = 0; j < JE; ++j) {
        const long long i = base + j * JT;
        p[j] = i < n55 ? (int)(i % nbf5) : 0;
        q[j] = i < n55 ? (int)(i / nbf5) : 0;
        sj[j] = sk[j] = 0.0;
    }
    if (JE == 1) {
        for (int l = l0; l < l1; ++l) {
            const T* B = bpq + n55 * l;
#pragma unroll
            for (int j = 0; j < JE; ++j) {
                const double v = B[p[j] + (long long)nbf5 * q[j]];
                sj[j] += (double)B[(long long)p[j] * (nbf5 + 1)] * (double)B[(long long)q[j] * (nbf5 + 1)];
                sk[j] += v * v;
            }
        }
    } else {
        for (int lb = l0; lb < l1; lb += JL) {
            const int nl = min(JL, l1 - lb);
            T v[JV][JE];
            auto fetch = [&](int h) {
#pragma unroll
                for (int k = 0; k < JV; ++k)
#pragma unroll
                    for (int j = 0; j < JE; ++j)
                        v[k][j] = h + k < nl ? bpq[n55 * (lb + h + k) + p[j] + (long long)nbf5 * q[j]] : T(0);
            };
            __syncthreads();  // the previous group's diagonals are read
            stage_diagonals<8>(bpq + n55 * lb, nbf5, 0, nbf5, nl, &sd[0][0], JD, 1);
            __syncthreads();
#pragma unroll
            for (int h = 0; h < JL; h += JV) {
                fetch(h);
#pragma unroll
                for (int k = 0; k < JV; ++k)
                    if (h + k < nl)
#pragma unroll
                        for (int j = 0; j < JE; ++j) {
                            const double x = (double)v[k][j];
                            sj[j] += sd[h + k][p[j]] * sd[h + k][q[j]];
                            sk[j] += x * x;
                        }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < JE; ++j) {
        const long long i = base + j * JT;
        if (i < n55) {
            part[(long long)c * 2 * n55 + i] = sj[j];
            part[(long long)c * 2 * n55 + n55 + i] = sk[j];
        }
    }
}

// The launch: grid (blocks, chunks).
template <class T>
void launch_partial(cudaStream_t st, const T* bpq, int nbf5, int naux, int lchunk, double* part) {
    const dim3 grid(blocks<T>(nbf5), (naux + lchunk - 1) / lchunk);
    if (per_thread<T>(nbf5) == 4) partial_kernel<T, 4><<<grid, JT, 0, st>>>(bpq, nbf5, naux, lchunk, part);
    else partial_kernel<T, 1><<<grid, JT, 0, st>>>(bpq, nbf5, naux, lchunk, part);
    count_launch();
}

}  // namespace jk
}  // namespace donof
