// Window-1 rotations over a hash-bucketed live set, several rotations per launch.
//
// The bucket hash h is GF(2)-linear (kernels_bucket.cuh): the partner P xor M of a
// term of bucket b lies in bucket b xor h(M), for every term alike.  For a block of
// K consecutive rotations with deltas h(M_1) .. h(M_K) the buckets therefore fall
// into the cosets of the span D of the deltas, and no term of a coset meets a term
// of another one within the block.  A CTA takes a coset (2^d buckets, d = dim D <=
// K), holds its terms in shared memory through the K rotations
// (_rotate_range! + _merge_spv!, spv_kernels.jl:146-177, 326-386, each with the
// same arithmetic and rounding as everywhere else), and writes the survivors to
// their buckets of the other bucket set.
//
// Within the block a rotation touches only the terms that anticommute with its
// generator: the others keep their value, and a value that has passed the strict
// filter once passes it again.  The filter is applied to every term only where
// values may not have passed it: at the first rotation of a call and after a
// channel (a block ends at a channel, which scales every survivor at its end).
//
// What bounds it: latency and instruction issue, and above a million terms the scattered
// reads and writes of short bucket runs (one sector a term).  A warp issues one instruction every 11 cycles
// (fixed latencies, shared memory), and twelve warps are what the resident sets leave
// room for.  Large sets: a warp per coset, no block barrier between rotations.  Small
// sets (an SM has a few cosets at most): a CTA per coset, whose chain of a rotation is
// shorter -- a thread per slot, or a batch per warp -- and whose larger resident set
// takes more rotations per launch.  The index over all resident terms is built once per
// block and pays from about three rotations on.
// Measured (one B200, whole calls, one rotation per launch before): 8 x 8 lattice,
// 3,520 rotations, up to 3.9e6 terms 154.9 -> 84 ms; 127-qubit graph, 6,504 rotations, up
// to 8e4 terms 43.4 -> 16.3 ms; 48 batched instances 60.1 -> 35 ms.  (A warp per coset
// everywhere: 109, 19.6 and 42.6; a CTA everywhere: 111, 16.2 and 38.4 with cosets of 512
// terms, 96, 18.9 and 38.4 with cosets of 900; the lattice at 95 then.)
#pragma once
#include "kernels_bucket.cuh"

namespace pp {

constexpr int BB_CAP = 32;                     // slots of a bucket
constexpr int BB_CAP_LOG = 5;
constexpr int BB_KMAX = 8;                     // rotations of a block at most
constexpr int BB_DMAX = 8;                     // dimension of a coset at most
constexpr int BB_MEMBERS = 1 << BB_DMAX;       // buckets of a coset at most
constexpr int BB_WARPS = 4;                    // warps of a CTA
constexpr unsigned BB_DEAD = 0x8000u;          // tag bit: the slot holds no live term

// Slots of the resident set and of its key index that T threads share: a warp (T = 32;
// twelve fit on an SM) or the CTA (T = 128; three).
template <int NW, int T>
__host__ __device__ constexpr int bb_slots() { return T == 32 ? (NW == 1 ? 448 : 288) : (NW == 1 ? 1920 : 1152); }
template <int T>
__host__ __device__ constexpr int bb_tab() { return T == 32 ? 1024 : 4096; }

constexpr int RS_QCAP = 160;                   // entries of a warp's queue of slots (31 + 4 * 32 at most)

// Shared memory of one resident set: coefficients, key words, index, tags.
template <int NW, int SLOTS, int TAB>
__host__ __device__ constexpr size_t rs_set_bytes() { return (size_t)SLOTS * (8 + 16 * NW + 2) + (size_t)TAB * 4; }
template <int NW, int T>
__host__ __device__ constexpr size_t bb_smem_bytes() {
    return 32 * BB_WARPS / T * rs_set_bytes<NW, bb_slots<NW, T>(), bb_tab<T>()>() + BB_WARPS * RS_QCAP * 2;
}

// One rotation as the steps use it: the generator's key words in 32-bit pieces
// (z low to high, then x), the planes its parity test reads with their masks, and
// cos / sin.
template <int NW>
struct RsGen {
    double cosv, sinv;
    unsigned g[4 * NW];
    unsigned mask[4 * NW];
    int plane[4 * NW];
    int np, ng, acol, delta, flags;
};

// Made by one warp (all lanes), a lane per plane.
template <int NW>
__device__ __forceinline__ void rs_gen(RsGen<NW> *o, const GenRec &g, int delta) {
    const int lane = threadIdx.x & 31;
    if (lane == 0) {
        o->cosv = g.cosv;
        o->sinv = g.sinv;
        o->ng = g.ng;
        o->acol = g.acol;
        o->delta = delta;
        o->flags = g.flags;
    }
    // plane p: the key's words z low to high, then x; its parity test (gx against z, gz
    // against x) reads only planes under a nonzero mask
    const int p = lane & (4 * NW - 1), q = p ^ (2 * NW);
    auto word = [&](int t) {
        const u64 v = t < 2 * NW ? g.gz[t >> 1] : g.gx[(t - 2 * NW) >> 1];
        return t & 1 ? (unsigned)(v >> 32) : (unsigned)v;
    };
    const unsigned mine = word(p), m = word(q);
    const unsigned on = __ballot_sync(0xffffffffu, lane < 4 * NW && m != 0);
    if (lane < 4 * NW) {
        o->g[p] = mine;
        if (m) {
            const int at = __popc(on & ((1u << lane) - 1u));
            o->plane[at] = p;
            o->mask[at] = m;
        }
    }
    if (lane == 0) o->np = __popc(on);
}

// The term in slot o of a bucket set (one-word keys: records at Z; two-word keys: three
// arrays), through L2 only: a bucket set is rewritten by every second launch, and a
// dependent launch may start before its predecessor's predecessor has ended, so its lines
// must not be served from an SM's L1.
template <int NW>
__device__ __forceinline__ void load_term(const u64 *Z, const u64 *X, const double *C, long long o, Key<NW> *k, double *c) {
    if constexpr (NW == 1) {
        const ulonglong2 *p = reinterpret_cast<const ulonglong2 *>(Z + o * BK_REC);
        const ulonglong2 a = __ldcg(p), b = __ldcg(p + 1);
        k->z[0] = a.x; k->x[0] = a.y;
        *c = __longlong_as_double((long long)b.x);
    } else {
        const ulonglong2 a = __ldcg(reinterpret_cast<const ulonglong2 *>(Z) + o);
        const ulonglong2 b = __ldcg(reinterpret_cast<const ulonglong2 *>(X) + o);
        k->z[0] = a.x; k->z[1] = a.y; k->x[0] = b.x; k->x[1] = b.y;
        *c = __ldcg(C + o);
    }
}
template <int NW>
__device__ __forceinline__ void store_term(u64 *Z, u64 *X, double *C, long long o, const Key<NW> &k, double c) {
    if constexpr (NW == 1) {
        ulonglong2 *p = reinterpret_cast<ulonglong2 *>(Z + o * BK_REC);
        p[0] = make_ulonglong2(k.z[0], k.x[0]);
        p[1] = make_ulonglong2((u64)__double_as_longlong(c), 0ull);      // the padding, too: a whole sector is written
    } else {
        store_key<NW>(Z, X, o, k);
        C[o] = c;
    }
}

// A key in 32-bit words: z low to high, then x.
template <int NW>
struct Key32 {
    unsigned w[4 * NW];
};

template <int NW>
__device__ __forceinline__ Key<NW> key_wide(const Key32<NW> &k) {
    Key<NW> o;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        o.z[w] = ((u64)k.w[2 * w + 1] << 32) | k.w[2 * w];
        o.x[w] = ((u64)k.w[2 * NW + 2 * w + 1] << 32) | k.w[2 * NW + 2 * w];
    }
    return o;
}

template <int NW>
__device__ __forceinline__ Key32<NW> key_narrow(const Key<NW> &k) {
    Key32<NW> o;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        o.w[2 * w] = (unsigned)k.z[w];
        o.w[2 * w + 1] = (unsigned)(k.z[w] >> 32);
        o.w[2 * NW + 2 * w] = (unsigned)k.x[w];
        o.w[2 * NW + 2 * w + 1] = (unsigned)(k.x[w] >> 32);
    }
    return o;
}

// 32-bit multiply-xor mix of a key: its low bits are the index position, its high
// 16 bits the fingerprint kept in the index entry.
template <int NW>
__device__ __forceinline__ unsigned rs_hash(const Key32<NW> &k) {
    unsigned h = k.w[0] * 0x9E3779B1u;
#pragma unroll
    for (int q = 1; q < 4 * NW; ++q) h = (h ^ k.w[q]) * (q & 1 ? 0x85EBCA77u : 0xC2B2AE3Du) + (h >> 17);
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 13;
    return h;
}

// A term set resident in shared memory: planes of 32-bit key words, coefficients,
// tags (local bucket, BB_DEAD), and an open-addressed index of every slot's key
// (entry: fingerprint << 16 | slot + 1).  Entries are never taken out: a dropped
// term's slot stays indexed, and the key's return finds and revives it.
template <int NW, int SLOTS, int TAB>
struct ResidentSet {
    double *c;
    unsigned *w;                    // [4 NW][SLOTS]
    unsigned *tab;                  // [TAB]
    unsigned short *tag;            // [SLOTS]

    __device__ __forceinline__ Key32<NW> key(int i) const {
        Key32<NW> k;
#pragma unroll
        for (int p = 0; p < 4 * NW; ++p) k.w[p] = w[p * SLOTS + i];
        return k;
    }
    __device__ __forceinline__ void put(int i, const Key32<NW> &k, double v, unsigned t) const {
#pragma unroll
        for (int p = 0; p < 4 * NW; ++p) w[p * SLOTS + i] = k.w[p];
        c[i] = v;
        tag[i] = (unsigned short)t;
    }
    __device__ __forceinline__ void insert(int i, unsigned h) const {
        const unsigned e = (h & 0xffff0000u) | (unsigned)(i + 1);
        unsigned p = h & (TAB - 1);
        for (int probe = 0; probe < TAB; ++probe) {
            if (atomicCAS(&tab[p], 0u, e) == 0u) return;
            p = (p + 1) & (TAB - 1);
        }
    }
    // slot of the key, or -1
    __device__ __forceinline__ int find(const Key32<NW> &k, unsigned h) const {
        unsigned p = h & (TAB - 1);
        for (int probe = 0; probe < TAB; ++probe) {
            const unsigned e = *(volatile unsigned *)&tab[p];
            if (e == 0) return -1;
            if (((e ^ h) & 0xffff0000u) == 0) {
                const int i = (int)(e & 0xffffu) - 1;
                unsigned d = 0;
#pragma unroll
                for (int q = 0; q < 4 * NW; ++q) d |= w[q * SLOTS + i] ^ k.w[q];
                if (d == 0) return i;
            }
            p = (p + 1) & (TAB - 1);
        }
        return -1;
    }
};

// What the steps read besides the set: the filters and, for batched instances,
// their angle tables and ends.
struct RsParams {
    FQuick strict;
    const DevFilter *strict_full;
    const DevFilter *local;
    bool local_on;
    const double *bcos, *bsin;
    const long long *bend;
    long long ninst;
    int ncol;
    DevState *S;
};

// Instance of a batched term, or -1 when it has ended before rotation r (or the tag
// is no instance).
template <int NW>
__device__ __forceinline__ long long rs_instance(const Key32<NW> &k, const RsParams &q, long long r) {
    const u64 t = ((u64)k.w[3 % (4 * NW)] << 32) | k.w[2 % (4 * NW)];     // z word 1
    if (t >= (u64)q.ninst) {
        flag_bounds(q.S, 11, (long long)t);
        return -1;
    }
    return r < q.bend[t] ? (long long)t : -1;
}

// Weight and X-weight caps of the strict filter on a key in 32-bit words (the rest of
// should_drop, spv_kernels.jl:64-79, is the coefficient's; a filter with other
// criteria is evaluated in full).  Without branches: the two keys of a pair are tested
// side by side, which a chain of short-circuit tests made 350 cycles of a step's 1,500.
template <int NW>
__device__ __forceinline__ bool rs_heavy(const RsParams &q, const Key32<NW> &k) {
    int wt = 0, xw = 0;
#pragma unroll
    for (int t = 0; t < 2 * NW; ++t) {
        wt += __popc(k.w[t] | k.w[2 * NW + t]);
        xw += __popc(k.w[2 * NW + t]);
    }
    return (wt > q.strict.wmax) | (xw > q.strict.xwmax);
}

template <int NW>
__device__ __forceinline__ bool rs_drop(const RsParams &q, const Key32<NW> &k, double absc) {
    if (q.strict.full) return should_drop<NW>(*q.strict_full, key_wide<NW>(k), absc);
    return (absc <= q.strict.thresh) | rs_heavy<NW>(q, k);
}

// <ket|.|ket> of dropped terms (EnergyCorrection), added up exactly, so that the sum does
// not depend on the order.  A value, scaled by the unit of the call (about the 2-norm of the
// entering set), is cut into whole multiples of 2^-30, 2^-62, 2^-94 and 2^-126: from 2^-70 to
// 2 in magnitude that is all of it, and the sums of all the terms that a set may hold (2^31)
// stay within 64 bits.  Other values, which are rare, go to words in global memory that
// cover every double: word k counts multiples of 2^(32 k - 1074).
static __device__ __noinline__ void rs_energy_rest(unsigned long long *word, int *flag, double v) {
    *flag = 1;
    const u64 b = (u64)__double_as_longlong(v);
    int e = (int)(b >> 52) & 0x7ff;
    u64 m = b & ((1ull << 52) - 1);
    if (e == 0x7ff) {                                          // an infinity or NaN
        atomicAdd(reinterpret_cast<double *>(word + BK_REST - 1), v);
        return;
    }
    if (e) {
        m |= 1ull << 52;
        --e;
    }
    const int k = e >> 5, o = e & 31;                          // v = m 2^(e - 1074), 53 + 31 bits from word k on
    const u64 part[3] = {(m << o) & 0xffffffffu, (m >> (32 - o)) & 0xffffffffu, o ? m >> (64 - o) : 0};
#pragma unroll
    for (int t = 0; t < 3; ++t)
        if (part[t]) atomicAdd(word + k + t, (unsigned long long)((b >> 63) ? 0 - part[t] : part[t]));
}

template <int NW>
struct RsEnergy {
    long long a[4];
    unsigned ket[2 * NW];
    double scale;
    unsigned long long *rest;
    int *rest_flag;
    __device__ __forceinline__ void add(const Key32<NW> &k, double v) {
        unsigned x = 0, s = 0;
#pragma unroll
        for (int t = 0; t < 2 * NW; ++t) {
            x |= k.w[2 * NW + t];
            s ^= k.w[t] & ket[t];
        }
        if (x) return;
        if (__popc(s) & 1) v = -v;
        double r = v * scale;
        if (!(fabs(r) >= 0x1p-70 && fabs(r) <= 2.0)) {
            if (v != 0.0) rs_energy_rest(rest, rest_flag, v);
            return;
        }
        const double g[4] = {0x1p30, 0x1p62, 0x1p94, 0x1p126}, u[4] = {0x1p-30, 0x1p-62, 0x1p-94, 0x1p-126};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const long long q = __double2ll_rn(r * g[t]);
            a[t] += q;
            r = __dsub_rn(r, (double)q * u[t]);            // exact: |q| < 2^53
        }
    }
};

// One rotation on one anticommuting slot i of the resident set.  Of two partners'
// slots (live or not) the lower runs it for both, so every slot has one writer in a
// step and no barrier is needed between the reads and the writes of a pair's
// coefficients.  A sin branch without a slot is appended at n0 + atomicAdd(*fresh).
// Returns the change of the live count in the low half and the sin branches appended
// (WindowCounters) in the high half.
// en: nullptr, or where dropped values are added up.
template <int NW, int SLOTS, int TAB, bool BATCH, bool ENERGY>
__device__ __forceinline__ int rs_pair(const ResidentSet<NW, SLOTS, TAB> &s, const RsGen<NW> &g, const RsParams &q, int i,
                                       int n0, int *fresh, int *full, long long r, RsEnergy<NW> *en) {
    const unsigned ti = s.tag[i];
    const double ci = s.c[i];
    const Key32<NW> k = s.key(i);
    Key32<NW> p;
#pragma unroll
    for (int t = 0; t < 4 * NW; ++t) p.w[t] = k.w[t] ^ g.g[t];
    const unsigned hp = rs_hash<NW>(p);
    const bool hk = rs_heavy<NW>(q, k), hq = rs_heavy<NW>(q, p);
    // phase of the sin branch of P (_rotate_range!, spv_kernels.jl:155-163); the
    // partner's has the opposite sign: k(P) + k(P xor M) = 0 mod 4, and k is odd
    int m1 = 0, nzp = 0, nzx = 0;
#pragma unroll
    for (int t = 0; t < 2 * NW; ++t) {
        m1 += __popc(g.g[2 * NW + t] & k.w[t]);
        nzp += __popc(p.w[t] & p.w[2 * NW + t]);
        nzx += __popc(k.w[t] & k.w[2 * NW + t]);
    }
    const int j = s.find(p, hp);
    const bool ai = !(ti & BB_DEAD);
    if (j >= 0 ? j < i : !ai) return 0;
    const unsigned tj = j >= 0 ? s.tag[j] : BB_DEAD;
    const bool aj = !(tj & BB_DEAD);
    if (!ai && !aj) return 0;
    const double cj = j >= 0 ? s.c[j] : 0.0;
    double cv = g.cosv, sv = g.sinv;
    if constexpr (BATCH) {
        const long long t = rs_instance<NW>(k, q, r);
        if (t < 0) return 0;
        cv = q.bcos[t * q.ncol + g.acol];
        sv = q.bsin[t * q.ncol + g.acol];
    }
    const double sgs = (nzp - g.ng - nzx + 2 * m1) & 2 ? sv : -sv;      // (k - 2) sin, k = 1 or 3
    const double si = __dmul_rn(sgs, ci);                        // lands on P xor M
    const double sj = __dmul_rn(-sgs, cj);                       // lands on P
    bool oki = ai, okj = aj;
    if (q.local_on) {
        oki = ai && !should_drop<NW>(*q.local, key_wide<NW>(p), fabs(si));
        okj = aj && !should_drop<NW>(*q.local, key_wide<NW>(k), fabs(sj));
    }
    // live value first, then the append (_try_merge!)
    double vi = __dmul_rn(ci, cv), vj = __dmul_rn(cj, cv);
    const double wi = __dadd_rn(vi, sj), wj = __dadd_rn(vj, si);
    vi = ai ? (okj ? wi : vi) : sj;
    vj = aj ? (oki ? wj : vj) : si;
    bool ki = ai | okj, kj = aj | oki;
    if (q.strict.full) {
        ki = ki && !should_drop<NW>(*q.strict_full, key_wide<NW>(k), fabs(vi));
        kj = kj && !should_drop<NW>(*q.strict_full, key_wide<NW>(p), fabs(vj));
    } else {
        ki &= !((fabs(vi) <= q.strict.thresh) | hk);
        kj &= !((fabs(vj) <= q.strict.thresh) | hq);
    }
    if constexpr (ENERGY) {
        if ((ai | okj) && !ki) en->add(k, vi);
        if ((aj | oki) && !kj) en->add(p, vj);
    }
    if (ki) s.c[i] = vi;
    if (ki != ai) s.tag[i] = (unsigned short)(ti ^ BB_DEAD);
    if (j >= 0) {
        if (kj) s.c[j] = vj;
        if (kj != aj) s.tag[j] = (unsigned short)(tj ^ BB_DEAD);
    } else if (kj) {
        const int o = n0 + atomicAdd(fresh, 1);
        if (o < SLOTS) {
            s.put(o, p, vj, (ti ^ (unsigned)g.delta) & ~BB_DEAD);
            __threadfence_block();
            s.insert(o, hp);
        } else {
            *full = 1;
        }
    }
    return (oki ? 0x10000 : 0) + (okj ? 0x10000 : 0) + (int)ki - (int)ai + (int)kj - (int)aj;
}

// One rotation over the n slots of a resident set that T threads share (T = 32: the
// calling warp; else the CTA; the set's earlier writes visible, a barrier of them all
// after it).  Each warp scans 128 slots at a time with the parity test alone (one
// 16-byte shared read per plane under the generator's mask), queues the
// anticommuting ones, and runs rs_pair on 32 of them at a time, so that the long path
// runs with full warps although only about a tenth of the terms take it.  Returns
// this thread's rs_pair sums.
template <int NW, int SLOTS, int TAB, int T, bool BATCH, bool ENERGY = false>
__device__ __forceinline__ int rs_step(const ResidentSet<NW, SLOTS, TAB> &s, const RsGen<NW> &g, const RsParams &q, int n,
                                       unsigned short *queue, int *fresh, int *full, long long r,
                                       RsEnergy<NW> *en = nullptr) {
    const int lane = threadIdx.x & 31, warp = T == 32 ? 0 : threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    int cnt = 0, out = 0;
    const int np = g.np;
    if constexpr (T > 32) {
        if (n <= T) {                                   // a thread per slot: no queue in the chain
            const int i = threadIdx.x;
            unsigned a = 0;
            if (i < n)
                for (int t = 0; t < np; ++t) a ^= s.w[g.plane[t] * SLOTS + i] & g.mask[t];
            return __popc(a) & 1 ? rs_pair<NW, SLOTS, TAB, BATCH, ENERGY>(s, g, q, i, n, fresh, full, r, en) : 0;
        }
    }
    const int p0 = g.plane[0] * SLOTS;
    const unsigned m0 = g.mask[0];
    for (int base = warp * 128;; base += (T / 32) * 128) {
        const bool more = base < n;                     // warp-uniform
        if (more) {
            const int i0 = base + 4 * lane;
            uint4 a = make_uint4(0u, 0u, 0u, 0u);
            if (i0 < n && np > 0) {
                const uint4 v = *reinterpret_cast<const uint4 *>(s.w + p0 + i0);
                a = make_uint4(v.x & m0, v.y & m0, v.z & m0, v.w & m0);
                for (int t = 1; t < np; ++t) {
                    const uint4 u = *reinterpret_cast<const uint4 *>(s.w + g.plane[t] * SLOTS + i0);
                    const unsigned m = g.mask[t];
                    a.x ^= u.x & m;
                    a.y ^= u.y & m;
                    a.z ^= u.z & m;
                    a.w ^= u.w & m;
                }
            }
            const unsigned b[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const bool on = (__popc(b[e]) & 1) != 0 && i0 + e < n;
                const unsigned m = __ballot_sync(0xffffffffu, on);
                if (on) queue[cnt + __popc(m & lt)] = (unsigned short)(i0 + e);
                cnt += __popc(m);
            }
            __syncwarp();
        }
        // 32 queued slots at a time (the rest, too, once the scan is done)
        while (cnt >= 32 || (!more && cnt > 0)) {
            const int take = min(cnt, 32);
            cnt -= take;
            if (lane < take) out += rs_pair<NW, SLOTS, TAB, BATCH, ENERGY>(s, g, q, queue[cnt + lane], n, fresh, full, r, en);
            __syncwarp();
        }
        if (!more) break;
    }
    return out;
}

// The strict filter over every live slot (terms whose values have not passed it yet);
// returns the change of the live count.
template <int NW, int SLOTS, int TAB, int T, bool BATCH, bool ENERGY = false>
__device__ __forceinline__ int rs_filter(const ResidentSet<NW, SLOTS, TAB> &s, const RsParams &q, int n, long long r,
                                         RsEnergy<NW> *en = nullptr) {
    int out = 0;
    for (int i = threadIdx.x & (T - 1); i < n; i += T) {
        const unsigned t = s.tag[i];
        if (t & BB_DEAD) continue;
        const Key32<NW> k = s.key(i);
        if constexpr (BATCH) {
            if (rs_instance<NW>(k, q, r) < 0) continue;
        }
        if (rs_drop<NW>(q, k, fabs(s.c[i]))) {
            s.tag[i] = (unsigned short)(t | BB_DEAD);
            out -= 1;
            if constexpr (ENERGY) en->add(k, s.c[i]);
        }
    }
    return out;
}

// A block of rotations [r0, r0 + K): the span of its deltas as a reduced basis
// (basis[q] has bit piv[q], no other basis vector has it; piv ascending), and each
// delta's coordinates (the bits at piv).
struct BbPlan {
    long long r0;
    int K, d, full, kprev, cur, bits, prechan;
    unsigned basis[BB_KMAX];
    int piv[BB_KMAX];
    int dl[BB_KMAX];
};

// Deltas of the generators [0, n): the bucket hash of each with all BK_ROWS rows (a
// layout of 2^bits buckets uses the low bits).
template <int NW>
__global__ void k_bb_deltas(const GenRec *gens, long long n, const u64 *rows, unsigned *out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[i] = bk_hash<NW>(gens[i].gz, gens[i].gx, rows, BK_ROWS);
}

// Modes of k_bb_block: plain; batched instances; adaptive sequences (blocks of one
// rotation, unfiltered: the terms that AdaptiveTruncation drops after the previous
// rotation -- |c| at most thr[r0] -- are dropped as they are loaded, a channel between
// the two (pl.prechan) is applied there, and the survivors' |c| are listed for the next
// threshold); plain with EnergyCorrection.
constexpr int BB_PLAIN = 0, BB_BATCH = 1, BB_ADAPT = 2, BB_ENERGY = 3;

// One block of rotations; input bucket set pl.cur, output set pl.cur ^ 1 (the input
// stays intact, so a block that does not fit -- a coset beyond the resident set, or
// an output bucket beyond BB_CAP -- is flagged and run again by the host, after a
// split or with fewer rotations).  Persistent grid; T threads take a coset at a time: a
// warp, whose rotations need no block barrier between them, or the CTA.
template <int NW, int MODE, int T>
__global__ void __launch_bounds__(32 * BB_WARPS, 3) k_bb_block(const __grid_constant__ BkArgs A,
                                                               const __grid_constant__ BbPlan pl) {
    constexpr bool BATCH = MODE == BB_BATCH;
    constexpr bool ADAPT = MODE == BB_ADAPT;
    constexpr bool ENERGY = MODE == BB_ENERGY;
    constexpr int SLOTS = bb_slots<NW, T>();
    constexpr int TAB = bb_tab<T>();
    constexpr int GROUPS = 32 * BB_WARPS / T;              // cosets a CTA works on at a time
    constexpr int ME = BB_MEMBERS / T;                     // members per thread at most
    static_assert(T == 32 || T == 32 * BB_WARPS, "a warp or the CTA per coset");
    static_assert(2 * 2 * BB_CAP <= SLOTS, "a block of one rotation always fits");
    static_assert(!BATCH || NW == 2, "batched instances use two-word keys");
    DevState *S = A.S;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __shared__ RsGen<NW> s_g[BB_KMAX];
    __shared__ int s_x[BB_MEMBERS];                        // a member's place in its coset
    __shared__ int s_cw[GROUPS][BB_MEMBERS];
    __shared__ unsigned short s_ow[GROUPS][BB_MEMBERS];
    __shared__ int s_fw[GROUPS][BB_KMAX + 1];              // fresh slots of each step, resident set full
    __shared__ int s_aw[GROUPS][BB_KMAX + 1][2];           // change of the live count, sin branches of each step
    __shared__ int s_scan[BB_WARPS + 1];
    __shared__ int s_tot[BB_KMAX][2], s_np, s_mx, s_over, s_err, s_pref, s_bad;
    __shared__ double s_thr;
    extern __shared__ __align__(16) unsigned char bbm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gt = tid & (T - 1), grp = tid / T;           // thread of the group, group of the CTA
    auto sync = [&]() {
        if constexpr (T == 32) __syncwarp();
        else __syncthreads();
    };
    ResidentSet<NW, SLOTS, TAB> set;
    unsigned char *mine = bbm + grp * rs_set_bytes<NW, SLOTS, TAB>();
    set.c = reinterpret_cast<double *>(mine);
    set.w = reinterpret_cast<unsigned *>(set.c + SLOTS);
    set.tab = set.w + 4 * NW * SLOTS;
    set.tag = reinterpret_cast<unsigned short *>(set.tab + TAB);
    unsigned short *queue = reinterpret_cast<unsigned short *>(bbm + GROUPS * rs_set_bytes<NW, SLOTS, TAB>()) + warp * RS_QCAP;
    int *scnt = s_cw[grp];
    unsigned short *soff = s_ow[grp];
    int *fresh = s_fw[grp], *full = &s_fw[grp][BB_KMAX];
    int (*acc)[2] = s_aw[grp];
    const int K = pl.K, d = pl.d, mem = 1 << d;
    const long long r0 = pl.r0;
    for (int j = warp; j < K; j += BB_WARPS) rs_gen<NW>(&s_g[j], A.gens[r0 + j], pl.dl[j]);
    if (tid < K) s_tot[tid][0] = s_tot[tid][1] = 0;
    const int last_flags = A.gens[r0 + K - 1].flags;
    if (tid == 0) { s_over = 0; s_bad = 0; s_mx = 0; s_np = 0; }
    for (int m = tid; m < mem; m += 32 * BB_WARPS) {
        unsigned b = 0;
        for (int e = 0; e < d; ++e)
            if ((m >> e) & 1) b ^= pl.basis[e];
        s_x[m] = (int)b;
    }
    for (int i = gt; i < TAB / 4; i += T) reinterpret_cast<uint4 *>(set.tab)[i] = make_uint4(0u, 0u, 0u, 0u);
    const DevParams &P = *A.P;
    RsParams q;
    q.strict = fquick(P.strict);
    q.strict_full = &P.strict;
    q.local = &P.local;
    q.local_on = P.local_active != 0;
    q.bcos = A.bcos;
    q.bsin = A.bsin;
    q.bend = A.bend;
    q.ninst = A.ninst;
    q.ncol = A.ncol;
    q.S = S;
    const bool do_chan = !ADAPT && (last_flags & GEN_CHANNEL) != 0 && P.chan_kind >= 0;
    const int cur = pl.cur;
    const int *CNT = cur ? A.cnt[1] : A.cnt[0];
    int *OCNT = cur ? A.cnt[0] : A.cnt[1];
    const u64 *Z = cur ? A.z[1] : A.z[0], *X = cur ? A.x[1] : A.x[0];
    const double *C = cur ? A.c[1] : A.c[0];
    u64 *OZ = cur ? A.z[0] : A.z[1], *OX = cur ? A.x[0] : A.x[1];
    double *OC = cur ? A.c[0] : A.c[1];
    // the previous block's outputs, records and error word are visible from here on
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (tid == 0) {
        s_err = *(volatile int *)&S->err;
        if constexpr (ADAPT) s_thr = *(const volatile double *)&A.thr[r0];
        // the early-merge rule of spv_evolve.jl:356-362 up to r0, from the previous
        // block's records (after a rotation every live value has passed the filter, so a
        // rotation inside a block that starts with an early merge drops nothing by it)
        const volatile BkRec *rec = A.rec;
        const long long nin = (long long)rec[r0].n_out;
        long long acap = rec[r0].acap;
        if (pl.kprev > 0) {
            const long long b = r0 - pl.kprev;
            long long nr[BB_KMAX];
#pragma unroll
            for (int e = 1; e < BB_KMAX; ++e) nr[e] = e < pl.kprev ? (long long)rec[b + e].n_out : 0;
            acap = rec[b + 1].acap;
            const long long np = (long long)rec[b + 1].np;
            if (rec[b + 1].pref && np > acap) acap = max(2 * acap, np);
#pragma unroll
            for (int e = 1; e < BB_KMAX; ++e)
                if (nr[e] > acap) acap = 2 * acap > nr[e] ? 2 * acap : nr[e];
        }
        const int pref = nin > acap ? 1 : 0;
        s_pref = pref;
        if (blockIdx.x == 0) {
            BkRec &me = A.rec[r0 + 1];
            me.n_in = nin;
            me.acap = acap;
            me.pref = pref;
            if (pref && !pl.full) me.np = (unsigned long long)nin;
        }
    }
    __syncthreads();
    if (s_err) return;
    const bool drop_first = ADAPT || (pl.full && s_pref);
    const double thr = ADAPT ? s_thr : 0.0;
    const long long nb = 1ll << pl.bits;
    if (pl.bits > A.bits_cap || d > pl.bits || d > BB_DMAX || K > BB_KMAX || r0 + K >= A.rec_len) {
        if (tid == 0) flag_bounds(S, 1, ((long long)pl.bits << 16) | d);
        return;
    }
    const long long ncos = nb >> d;
    int tot_out = 0, tot_cre = 0;                          // thread j < K of the group: rotation r0 + j
    int tot_np = 0, mx = 0;                                // (tot_np: the group's thread 0)
    bool over = false;
    RsEnergy<NW> en = {};
    if constexpr (ENERGY) {
        en.scale = A.escale;
        en.rest = A.rest + (r0 + 1) * BK_REST;
        en.rest_flag = &A.rec[r0 + 1].rest;
#pragma unroll
        for (int t = 0; t < 2 * NW; ++t) en.ket[t] = (unsigned)(P.ket[t >> 1] >> (32 * (t & 1)));
    }
    // one barrier has to follow a step's counts before they are read: with a warp per
    // coset they stay in registers, with a CTA they meet in acc[j]
    auto counted = [&](int out, int j) {                   // call with the whole group; returns after the barrier
        out = __reduce_add_sync(0xffffffffu, out);
        if constexpr (T == 32) {
            sync();
            return out;
        } else {
            if (lane == 0 && out) {
                const int dn = (int)(short)(out & 0xffff);
                atomicAdd(&acc[j][0], dn);
                atomicAdd(&acc[j][1], (out - dn) >> 16);
            }
            sync();
            return 0;
        }
    };
    for (long long cs = (long long)blockIdx.x * GROUPS + grp; cs < ncos; cs += (long long)gridDim.x * GROUPS) {
        // ---- the coset's buckets and their places in the resident set
        int total = 0;
        unsigned rep = (unsigned)cs;                       // member m is bucket rep ^ s_x[m]
        for (int e = 0; e < d; ++e) {
            const int p = pl.piv[e];
            rep = ((rep >> p) << (p + 1)) | (rep & ((1u << p) - 1u));
        }
        {
            int nm[ME];
#pragma unroll
            for (int e = 0; e < ME; ++e) {
                const int m = T * e + gt;
                nm[e] = 0;
                if (m < mem) {
                    const unsigned b = rep ^ (unsigned)s_x[m];
                    if (b < nb) nm[e] = __ldcg(CNT + b);
                    else { flag_bounds(S, 3, b); s_bad = 1; }
                }
            }
            if (gt <= BB_KMAX) {
                fresh[gt] = 0;                             // and *full
                acc[gt][0] = acc[gt][1] = 0;
            }
#pragma unroll
            for (int e = 0; e < ME; ++e) {
                if (T * e < mem) {                         // uniform
                    if (nm[e] < 0 || nm[e] > BB_CAP) { flag_bounds(S, 4, nm[e]); s_bad = 1; nm[e] = 0; }
                    int o, sum;
                    if constexpr (T == 32) {
                        const int inc = warp_incl_scan(nm[e], OpSum());
                        o = total + inc - nm[e];
                        sum = __shfl_sync(0xffffffffu, inc, 31);
                    } else {
                        o = total + block_excl_scan<T>(nm[e], 0, OpSum(), s_scan, &sum);
                    }
                    const int m = T * e + gt;
                    if (m < mem) {
                        soff[m] = (unsigned short)o;
                        scnt[m] = 0;
                        if (o + nm[e] <= SLOTS)            // each slot's bucket
                            for (int t = 0; t < nm[e]; ++t) set.tag[o + t] = (unsigned short)m;
                    }
                    total += sum;
                }
            }
            sync();
        }
        if (total > SLOTS) { over = true; continue; }      // uniform
        // ---- load and index, LU terms a thread in flight
        constexpr int LU = 2;
        int dropped = 0;
        for (int b0 = 0; b0 < total; b0 += LU * T) {
            Key<NW> kk[LU];
            double cc[LU];
            int lb[LU];
#pragma unroll
            for (int u = 0; u < LU; ++u) {
                const int i = b0 + u * T + gt;
                if (i < total) {
                    lb[u] = set.tag[i];
                    const long long o = ((long long)(rep ^ (unsigned)s_x[lb[u]]) << BB_CAP_LOG) + (i - soff[lb[u]]);
                    load_term<NW>(Z, X, C, o, &kk[u], &cc[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < LU; ++u) {
                const int i = b0 + u * T + gt;
                if (i < total) {
                    const Key32<NW> k = key_narrow<NW>(kk[u]);
                    bool dead = false;
                    if constexpr (ADAPT) {
                        dead = fabs(cc[u]) <= thr;
                        if (pl.prechan && !dead) cc[u] = __dmul_rn(cc[u], channel_factor<NW>(P, kk[u]));
                    } else if (drop_first) {
                        dead = rs_drop<NW>(q, k, fabs(cc[u]));
                        if constexpr (BATCH) dead = dead && rs_instance<NW>(k, q, r0) >= 0;
                        if constexpr (ENERGY) { if (dead) en.add(k, cc[u]); }
                    }
                    dropped += dead ? 1 : 0;
                    set.put(i, k, cc[u], (unsigned)lb[u] | (dead ? BB_DEAD : 0u));
                    set.insert(i, rs_hash<NW>(k));
                }
            }
        }
        int alive = total;
        if (drop_first) {
            dropped = __reduce_add_sync(0xffffffffu, dropped);
            if constexpr (T == 32) {
                alive -= dropped;
            } else {
                if (lane == 0 && dropped) atomicAdd(&acc[BB_KMAX][0], dropped);
                sync();
                alive -= acc[BB_KMAX][0];
            }
            if (gt == 0) tot_np += alive;
        }
        sync();
        // ---- the K rotations
        int n = total;
        for (int j = 0; j < K; ++j) {
            int out = counted(rs_step<NW, SLOTS, TAB, T, BATCH, ENERGY>(set, s_g[j], q, n, queue, &fresh[j], full, r0 + j, &en), j);
            n = min(n + fresh[j], SLOTS);
            if (j == 0 && pl.full) out += counted(rs_filter<NW, SLOTS, TAB, T, BATCH, ENERGY>(set, q, n, r0, &en), 0);
            int dn, cre;
            if constexpr (T == 32) {
                dn = (int)(short)(out & 0xffff);
                cre = (out - dn) >> 16;
            } else {
                dn = acc[j][0];
                cre = acc[j][1];
            }
            alive += dn;
            if (gt == j) { tot_cre += cre; tot_out += alive; }
        }
        // ---- the survivors to their buckets of the output set, the index cleared
        if (*full) {
            over = true;
        } else {
            long long vat = 0;                             // adaptive: where this coset's values go
            if constexpr (ADAPT) {
                static_assert(T == 32, "adaptive sequences use a warp per coset");
                if (lane == 0) vat = (long long)atomicAdd(&A.rec[r0 + 1].nval, (unsigned long long)alive);
                vat = __shfl_sync(0xffffffffu, vat, 0);
            }
            for (int base = T == 32 ? 0 : warp * 32; base < n; base += T) {
                const int i = base + lane;
                const unsigned t = i < n ? set.tag[i] : BB_DEAD | 0x7fffu;
                const bool live = !(t & BB_DEAD);
                if constexpr (ADAPT) {
                    const unsigned m = __ballot_sync(0xffffffffu, live);
                    const long long o = vat + __popc(m & ((1u << lane) - 1u));
                    if (live && o < A.vals_cap) A.vals[o] = fabs(set.c[i]);
                    vat += __popc(m);
                }
                const int lb = (int)(t & 0xff);
                const unsigned seg = bk_segment((int)(t & 0x7fffu), lane);
                const int po = bk_claim(scnt, lb, live, seg, lane);
                if (live && po < BB_CAP && lb < mem) {
                    const Key<NW> kw = key_wide<NW>(set.key(i));
                    double v = set.c[i];
                    bool ch = do_chan;
                    if constexpr (BATCH) ch = ch && rs_instance<NW>(set.key(i), q, r0 + K - 1) >= 0;
                    if (ch) v = __dmul_rn(v, channel_factor<NW>(P, kw));
                    const long long o = ((long long)(rep ^ (unsigned)s_x[lb]) << BB_CAP_LOG) + po;
                    store_term<NW>(OZ, OX, OC, o, kw, v);
                }
            }
        }
        for (int i = gt; i < TAB / 4; i += T) reinterpret_cast<uint4 *>(set.tab)[i] = make_uint4(0u, 0u, 0u, 0u);
        sync();
        for (int m = gt; m < mem; m += T) {
            const int c = scnt[m];
            const unsigned b = rep ^ (unsigned)s_x[m];
            if (b < nb) OCNT[b] = min(c, BB_CAP);
            mx = max(mx, c);
        }
        sync();
    }
    if constexpr (ENERGY) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            for (int o = 16; o > 0; o >>= 1) en.a[t] += __shfl_xor_sync(0xffffffffu, en.a[t], o);
            if (lane == 0 && en.a[t]) atomicAdd(&A.rec[r0 + 1].energy[t], (unsigned long long)en.a[t]);
        }
    }
    // ---- the block's totals
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (gt < K) {
        atomicAdd(&s_tot[gt][0], tot_out);
        atomicAdd(&s_tot[gt][1], tot_cre);
    }
    if (lane == 0) {
        atomicMax(&s_mx, mx);
        atomicAdd(&s_np, tot_np);
        if (over || mx > BB_CAP) atomicOr(&s_over, (over ? 2 : 0) | (mx > BB_CAP ? 1 : 0));
    }
    __syncthreads();
    if (tid < K) {
        atomicAdd(&A.rec[r0 + tid + 1].n_out, (unsigned long long)s_tot[tid][0]);
        atomicAdd(&A.rec[r0 + tid + 1].created, (unsigned long long)s_tot[tid][1]);
    }
    if (tid == 0) {
        if (drop_first) atomicAdd(&A.rec[r0 + 1].np, (unsigned long long)s_np);
        atomicMax(&A.rec[r0 + K].maxcnt, s_mx);
        if (s_over) {
            atomicOr(&S->bk_over, s_over);                  // 1: a bucket overflowed, 2: a coset beyond the resident set
            atomicMin(&S->bk_fail, r0);
            atomicOr(&S->err, ERR_OVERFLOW);
        }
        if (s_bad) atomicOr(&S->err, ERR_BOUNDS);
    }
}

}  // namespace pp
