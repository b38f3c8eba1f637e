// Stable sort of (z, x, c) records by the (z, x) key: a sample sort.
//
// Records are ranked by (key, position), which no two share, so the sort is stable
// and equal keys cannot make a bucket large:
//   k_ss_sample  S = 8 evenly strided records per bucket;
//   k_ss_rank    the rank of each sample, by counting over blocks of 256 x 256;
//   k_ss_split   every 8th sample in rank order is a splitter;
//   k_ss_scatter each record to its bucket (binary search over the splitters in
//                shared memory; a CTA takes a range of every bucket it meets from one
//                atomic; the order inside a bucket does not matter);
//   k_ss_sort    one CTA per bucket: bitonic sort of an index in shared memory, and
//                the records to their place in the output.
// Two passes over the records instead of one per 8-bit digit on which the keys differ
// (24 to 32 passes of five launches each for 64 and 128 qubits): the digit passes were
// bound by their launches up to 10^5 records and by uncoalesced writes above.
// Bound by latency below 10^5 records (five launches, each a few microseconds), by the
// bitonic sort's shared-memory traffic above.  Measured (one B200, with the digit passes
// before): 1.5e6 one-word records 0.80 -> 0.42 ms, 7e4 two-word records 1.4 -> 0.1 ms,
// a 7 x 9 lattice layer by layer (a sort per layer, up to 3e5 records) 15.4 -> 10.8 ms.
// Above SS_MAX the buckets would be too large for one CTA's shared memory; there, and
// when a bucket is beyond its slots (a flag; the source is written by k_ss_sort only),
// the caller sorts by digits.
#pragma once
#include "kernels_general.cuh"

namespace pp {

constexpr int SS_CAP = 4096;                   // slots of a bucket at most (half of it for small means: three CTAs per SM)
constexpr int SS_MAXB = 2048;                  // buckets at most
constexpr int SS_SAMPLES = 16384;              // samples at most
constexpr long long SS_MAX = 2200000;          // records at most (2048 buckets of 1,075 on average)
constexpr int SS_THREADS = 512;                // scatter
constexpr int SS_ITEMS = 4;
constexpr int SSS_THREADS = 512;               // bucket sort

template <int NW>
__device__ __forceinline__ bool ss_less(const Key<NW> &a, unsigned ia, const Key<NW> &b, unsigned ib) {
#pragma unroll
    for (int w = NW - 1; w >= 0; --w)
        if (a.z[w] != b.z[w]) return a.z[w] < b.z[w];
#pragma unroll
    for (int w = NW - 1; w >= 0; --w)
        if (a.x[w] != b.x[w]) return a.x[w] < b.x[w];
    return ia < ib;
}

// Sample i: record floor((i + 1/2) n / S); clears the ranks and the bucket counts.
template <int NW>
__global__ void k_ss_sample(const u64 *Z, const u64 *X, long long n, int S, Key<NW> *key, unsigned *pos, int *rank,
                            int *cnt, int nbk, int *over) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < S) {
        long long p = (long long)(((double)i + 0.5) * (double)n / (double)S);
        if (p >= n) p = n - 1;
        key[i] = load_key<NW>(Z, X, p);
        pos[i] = (unsigned)p;
        rank[i] = 0;
    }
    if (i < nbk) cnt[i] = 0;
    if (i == 0) *over = 0;
}

constexpr int SSR = 256;
template <int NW>
__global__ void __launch_bounds__(SSR) k_ss_rank(const Key<NW> *key, const unsigned *pos, int S, int *rank) {
    __shared__ Key<NW> sk[SSR];
    __shared__ unsigned sp[SSR];
    const int o = blockIdx.y * SSR + threadIdx.x, i = blockIdx.x * SSR + threadIdx.x;
    if (o < S) { sk[threadIdx.x] = key[o]; sp[threadIdx.x] = pos[o]; }
    __syncthreads();
    if (i >= S) return;
    const Key<NW> k = key[i];
    const unsigned p = pos[i];
    const int m = min(SSR, S - (int)blockIdx.y * SSR);
    int r = 0;
    for (int t = 0; t < m; ++t) r += ss_less<NW>(sk[t], sp[t], k, p) ? 1 : 0;
    if (r) atomicAdd(&rank[i], r);
}

// Splitter j: the sample of rank (j + 1) os - 1 (the last record of bucket j's samples).
template <int NW>
__global__ void k_ss_split(const Key<NW> *key, const unsigned *pos, const int *rank, int S, int os, int nbk, Key<NW> *skey,
                           unsigned *spos) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= S) return;
    const int r = rank[i] + 1;
    if (r % os == 0 && r / os < nbk) {
        skey[r / os - 1] = key[i];
        spos[r / os - 1] = pos[i];
    }
}

template <int NW>
__host__ __device__ constexpr size_t ss_scatter_smem(int nbk) { return (size_t)nbk * (16 * NW + 4 + 8); }

template <int NW>
__global__ void __launch_bounds__(SS_THREADS) k_ss_scatter(const u64 *Z, const u64 *X, const double *C, long long n,
                                                           const Key<NW> *skey, const unsigned *spos, int nbk, int *cnt,
                                                           u64 *BZ, u64 *BX, double *BC, unsigned *BP, int cap, int *over) {
    extern __shared__ __align__(16) unsigned char ssm[];
    Key<NW> *sk = reinterpret_cast<Key<NW> *>(ssm);
    unsigned *sp = reinterpret_cast<unsigned *>(sk + nbk);
    int *hist = reinterpret_cast<int *>(sp + nbk);
    int *base = hist + nbk;
    const int tid = threadIdx.x;
    for (int j = tid; j < nbk; j += SS_THREADS) {
        if (j < nbk - 1) { sk[j] = skey[j]; sp[j] = spos[j]; }
        hist[j] = 0;
    }
    __syncthreads();
    const long long b0 = (long long)blockIdx.x * SS_THREADS * SS_ITEMS;
    Key<NW> k[SS_ITEMS];
    double c[SS_ITEMS];
    int bk[SS_ITEMS], at[SS_ITEMS];
#pragma unroll
    for (int u = 0; u < SS_ITEMS; ++u) {
        const long long i = b0 + u * SS_THREADS + tid;
        bk[u] = -1;
        if (i < n) {
            k[u] = load_key<NW>(Z, X, i);
            c[u] = C[i];
        }
    }
#pragma unroll
    for (int u = 0; u < SS_ITEMS; ++u) {
        const long long i = b0 + u * SS_THREADS + tid;
        if (i < n) {
            // the first bucket whose splitter is not below the record
            int lo = 0, hi = nbk - 1;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (ss_less<NW>(sk[mid], sp[mid], k[u], (unsigned)i)) lo = mid + 1;
                else hi = mid;
            }
            bk[u] = lo;
            at[u] = atomicAdd(&hist[lo], 1);
        }
    }
    __syncthreads();
    for (int j = tid; j < nbk; j += SS_THREADS) base[j] = hist[j] ? atomicAdd(&cnt[j], hist[j]) : 0;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < SS_ITEMS; ++u) {
        if (bk[u] < 0) continue;
        const int p = base[bk[u]] + at[u];
        if (p >= cap) { *over = 1; continue; }
        const long long o = (long long)bk[u] * cap + p;
        store_key<NW>(BZ, BX, o, k[u]);
        BC[o] = c[u];
        BP[o] = (unsigned)(b0 + u * SS_THREADS + tid);
    }
}

// Shared memory of a bucket of at most cap records (a power of two).
template <int NW>
__host__ __device__ constexpr size_t ss_sort_smem(int cap) { return (size_t)cap * (16 * NW + 8 + 4 + 2); }

// Bucket blockIdx.x of at most cap records (cap: a power of two) sorted into the
// output at the sum of the earlier buckets' counts.  cnt == nullptr: the n records of
// (BZ, BX, BC) are one bucket, in position order.
template <int NW>
__global__ void __launch_bounds__(SSS_THREADS) k_ss_sort(const u64 *BZ, const u64 *BX, const double *BC, const unsigned *BP,
                                                         const int *cnt, int n, int cap, const int *over, u64 *Z, u64 *X,
                                                         double *C, long long ocap) {
    extern __shared__ __align__(16) unsigned char ssm[];
    constexpr int T = SSS_THREADS;
    u64 *kz = reinterpret_cast<u64 *>(ssm);                       // [NW][cap]
    u64 *kx = kz + (size_t)NW * cap;
    double *sc = reinterpret_cast<double *>(kx + (size_t)NW * cap);
    unsigned *sp = reinterpret_cast<unsigned *>(sc + cap);
    unsigned short *perm = reinterpret_cast<unsigned short *>(sp + cap);
    __shared__ int s_red[T / 32];
    const int tid = threadIdx.x, b = blockIdx.x;
    if (over && *over) return;
    int m = n;
    long long off = 0, src = 0;
    if (cnt) {
        m = cnt[b];
        int s = 0;
        for (int j = tid; j < b; j += T) s += cnt[j];
        s = __reduce_add_sync(0xffffffffu, s);
        if ((tid & 31) == 0) s_red[tid >> 5] = s;
        __syncthreads();
        for (int w = 0; w < T / 32; ++w) off += s_red[w];
        src = (long long)b * cap;
    }
    if (m < 0 || m > cap || off + m > ocap) return;               // (flagged as over, or an output that cannot hold it)
    int P = 1;
    while (P < m) P <<= 1;
    for (int i = tid; i < P; i += T) {
        perm[i] = (unsigned short)i;
        if (i < m) {
            const Key<NW> k = load_key<NW>(BZ, BX, src + i);
#pragma unroll
            for (int w = 0; w < NW; ++w) { kz[w * cap + i] = k.z[w]; kx[w * cap + i] = k.x[w]; }
            sc[i] = BC[src + i];
            sp[i] = BP ? BP[src + i] : (unsigned)i;
        }
    }
    __syncthreads();
    // slots at or above m sort behind every record, in slot order
    auto after = [&](int u, int v) {                              // record u belongs after record v
        if (u >= m || v >= m) return u > v;
#pragma unroll
        for (int w = NW - 1; w >= 0; --w) {
            const u64 a = kz[w * cap + u], c = kz[w * cap + v];
            if (a != c) return a > c;
        }
#pragma unroll
        for (int w = NW - 1; w >= 0; --w) {
            const u64 a = kx[w * cap + u], c = kx[w * cap + v];
            if (a != c) return a > c;
        }
        return sp[u] > sp[v];
    };
    for (int k = 2; k <= P; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int q = tid; q < P / 2; q += T) {
                const int i = ((q & ~(j - 1)) << 1) | (q & (j - 1)), l = i | j;
                const int u = perm[i], v = perm[l];
                if (after(u, v) == ((i & k) == 0)) {
                    perm[i] = (unsigned short)v;
                    perm[l] = (unsigned short)u;
                }
            }
            // pairs less than 32 apart stay within the 64 slots of a warp's 32 threads
            if (j > 32) __syncthreads();
            else __syncwarp();
        }
        __syncthreads();
    }
    for (int i = tid; i < m; i += T) {
        const int u = perm[i];
        Key<NW> k;
#pragma unroll
        for (int w = 0; w < NW; ++w) { k.z[w] = kz[w * cap + u]; k.x[w] = kx[w * cap + u]; }
        store_key<NW>(Z, X, off + i, k);
        C[off + i] = sc[u];
    }
}

}  // namespace pp
