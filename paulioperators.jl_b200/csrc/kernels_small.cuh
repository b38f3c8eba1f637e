// Window-1 rotations of a small live set in one CTA.  While the live set holds at
// most small_cap<NW>() terms, one launch runs rotation after rotation with the
// whole set in shared memory, instead of a launch per block of rotations, whose
// fixed latency dominates small sets.  It is the same sequence
// (spv_evolve.jl:352-385, spv_kernels.jl:146-177, 326-386) with the same per-term
// arithmetic (the resident set and its steps of kernels_block.cuh), so results are
// bit-identical to the other paths:
//   - the set and the index of its keys stay from rotation to rotation; a rotation
//     touches the anticommuting terms only.  Dropped terms leave dead slots, and when
//     the slots run out the live terms are moved together and indexed anew;
//   - where values may not have passed the strict filter yet (the first rotation, and
//     the one after a channel) it is applied to every term: before the rotation when
//     it starts with an early merge (n > acap), else after it;
//   - a channel scales every live term after its rotation;
//   - counters and WindowCounters records as the other paths write them.
// One barrier per rotation (two at a channel).  The set is sorted once, when the launch ends (bitonic
// over an index array; keys are distinct), and <ket|O|ket> of a measured last rotation
// is reduced on the sorted set.  The launch stops when the set outgrows small_cap or
// the call's rotations are done, and leaves the live set dense and sorted in the other
// buffer set.  It does not handle local truncation, corrections or batched instances;
// the host launches it only without them.  No waits: every barrier is in uniform
// control flow, every loop is bounded by the rotation count, the set size or the table
// size.
// Bound by the latency of a rotation's chain: parity test, index look-up, two products
// and a sum, filter, barrier -- about 1,700 cycles at 170 terms.  Measured (one B200,
// with a table and a copy of the set made anew every rotation before): 20-qubit chain,
// 312 rotations of 170 terms on average, 458 -> 302 us of kernel; the first 1,444
// rotations of a 127-qubit circuit 2.07 -> 1.15 ms.
#pragma once
#include "kernels_struct.cuh"
#include "kernels_block.cuh"

namespace pp {

constexpr int SM_THREADS = 512;                   // a thread per slot up to 512 (256: 6 % slower on a 20-qubit chain)

template <int NW>
__host__ __device__ constexpr int small_cap() { return NW == 1 ? 2048 : 1024; }

// a resident set of 2C slots (a rotation at most doubles the set), the warps' queues
template <int NW>
constexpr size_t small_smem() {
    constexpr int C = small_cap<NW>();
    return rs_set_bytes<NW, 2 * C, 4 * C>() + (SM_THREADS / 32) * RS_QCAP * 2;
}

template <int NW>
__global__ void __launch_bounds__(SM_THREADS, 1) k_small_run(Bufs B) {
    constexpr int C = small_cap<NW>();
    constexpr int SLOTS = 2 * C, TAB = 4 * C;
    constexpr int T = SM_THREADS;
    static_assert(SLOTS < 0x8000, "slots in 16 bits");
    DevState *S = B.S;
    __shared__ int s_go, s_full;
    __shared__ int s_cnt[3][3];                    // of rotation r in r % 3: fresh slots, change of the live count, sin branches
    __shared__ int s_scan[T / 32 + 1];
    __shared__ double s_red[T / 32];
    __shared__ __align__(16) GenRec gs[2];         // generators on their way in (the last warp's)
    __shared__ RsGen<NW> rg[3];                    // of this rotation and the next two, r % 3
    static_assert(sizeof(GenRec) % 16 == 0, "generator records copy in 16-byte pieces");
    constexpr int GQ = (int)(sizeof(GenRec) / 16);
    extern __shared__ __align__(16) unsigned char smr[];
    ResidentSet<NW, SLOTS, TAB> set;
    set.c = reinterpret_cast<double *>(smr);
    set.w = reinterpret_cast<unsigned *>(set.c + SLOTS);
    set.tab = set.w + 4 * NW * SLOTS;
    set.tag = reinterpret_cast<unsigned short *>(set.tab + TAB);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned short *queue = set.tag + SLOTS + warp * RS_QCAP;

    if (tid == 0) {
        s_go = (S->err == 0 && S->rot < S->rot_end && S->n <= C) ? 1 : 0;
        s_full = 0;
    }
    if (tid < 9) (&s_cnt[0][0])[tid] = 0;
    __syncthreads();
    if (!s_go) return;
    const DevParams &P = *B.P;
    RsParams q;
    memset(&q, 0, sizeof q);
    q.strict = fquick(P.strict);
    q.strict_full = &P.strict;
    q.local = &P.local;
    q.S = S;
    const u64 ket[2] = {P.ket[0], P.ket[1]};
    const int chan_kind = P.chan_kind;
    const int cur = S->cur;
    int n = (int)S->n, alive = n;                  // slots in use, live terms
    auto clear_index = [&]() {
        for (int i = tid; i < TAB / 4; i += T) reinterpret_cast<uint4 *>(set.tab)[i] = make_uint4(0u, 0u, 0u, 0u);
    };
    clear_index();
    __syncthreads();
    {
        // the live set: dense, or the segment table of the last multi-kernel merge
        const u64 *Z = B.z[cur], *X = B.x[cur];
        const double *Cc = B.c[cur];
        const bool dense = S->seg_dense != 0;
        const int nseg = (int)S->nseg;
        for (int i = tid; i < n; i += T) {
            long long p = i;
            if (!dense) {
                int lo = 0, hi = nseg - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (B.soff[mid] <= i) lo = mid; else hi = mid - 1;
                }
                p = (long long)B.sphys[lo] + (i - B.soff[lo]);
            }
            if (p < 0 || p >= B.cap) { atomicOr(&S->err, ERR_BOUNDS); p = 0; }
            const Key32<NW> k = key_narrow<NW>(load_key<NW>(Z, X, p));
            set.put(i, k, Cc[p], 0u);
            set.insert(i, rs_hash<NW>(k));
        }
    }
    long long rot = S->rot;
    const long long rot0 = rot, rot_end = S->rot_end;
    // the last warp copies generators in two rotations ahead and prepares them one
    // rotation later, while the others work; a barrier publishes them
    const bool feeder = warp == T / 32 - 1;
    auto fetch_gen = [&](long long r) {
        if (r < rot_end && lane < GQ)
            cp_async16(reinterpret_cast<char *>(&gs[r & 1]) + 16 * lane, reinterpret_cast<const char *>(B.gens + r) + 16 * lane);
        cp_async_commit();
    };
    auto make_gen = [&](long long r) {                // copied in before
        cp_async_wait_all();
        __syncwarp();
        if (r < rot_end) rs_gen<NW>(&rg[(r - rot0) % 3], gs[r & 1], 0);
        __syncwarp();
    };
    if (feeder)
        for (int k = 0; k < 3; ++k) {
            fetch_gen(rot + k);
            if (k < 2) make_gen(rot + k);
        }
    long long acap = S->acap_logical;
    long long created = 0, merge_out = 0, live_in = 0;
    int early = 0, peak = 0;
    bool measure_last = false, full = true;
    // the change of the live count and the sin branches of a pass, added up in s_cnt[k]
    auto count = [&](int out, int k) {
        if (__any_sync(0xffffffffu, out != 0)) {
            out = __reduce_add_sync(0xffffffffu, out);
            if (lane == 0) {
                const int dn = (int)(short)(out & 0xffff);
                if (dn) atomicAdd(&s_cnt[k][1], dn);
                if (out - dn) atomicAdd(&s_cnt[k][2], (out - dn) >> 16);
            }
        }
    };

    __syncthreads();
    for (int k3 = 0;; k3 = k3 == 2 ? 0 : k3 + 1) {
        const RsGen<NW> &g = rg[k3];
        if (feeder) {
            // the next rotation's counters start from zero (their last readers have passed a barrier)
            if (lane < 3) s_cnt[k3 == 2 ? 0 : k3 + 1][lane] = 0;
            make_gen(rot + 2);
            fetch_gen(rot + 3);
        }
        const bool pref = alive > acap;
        const int flags = g.flags;
        const bool do_chan = (flags & GEN_CHANNEL) != 0 && chan_kind >= 0;
        measure_last = (flags & GEN_MEASURE) != 0;
        // room for every live term's sin branch: else the live terms are moved together
        if (n + alive > SLOTS) {
            unsigned short *list = reinterpret_cast<unsigned short *>(set.tab);
            int m = 0;
            for (int base = 0; base < n; base += T) {
                const int i = base + tid;
                const int on = i < n && !(set.tag[i] & BB_DEAD) ? 1 : 0;
                int tot;
                const int o = m + block_excl_scan<T>(on, 0, OpSum(), s_scan, &tot);
                if (on) list[o] = (unsigned short)i;
                m += tot;
            }
            __syncthreads();
            for (int base = 0; base < m; base += T) {         // a term's new slot is never above its old one
                const int i = base + tid;
                Key32<NW> k;
                double v = 0.0;
                if (i < m) { k = set.key(list[i]); v = set.c[list[i]]; }
                __syncthreads();
                if (i < m) set.put(i, k, v, 0u);
                __syncthreads();
            }
            clear_index();
            __syncthreads();
            for (int i = tid; i < m; i += T) set.insert(i, rs_hash<NW>(set.key(i)));
            n = m;
            __syncthreads();
        }
        const int n_in = alive;
        long long np = n_in;
        if (full && pref) {
            count(rs_filter<NW, SLOTS, TAB, T, false>(set, q, n, rot), k3);
            __syncthreads();
            np = n_in + s_cnt[k3][1];
            __syncthreads();                       // read by every thread before the rotation adds to it
        }
        const int out = rs_step<NW, SLOTS, TAB, T, false>(set, g, q, n, queue, &s_cnt[k3][0], &s_full, rot);
        count(out, k3);
        __syncthreads();
        n = min(n + s_cnt[k3][0], SLOTS);
        if (full && !pref) {
            count(rs_filter<NW, SLOTS, TAB, T, false>(set, q, n, rot), k3);
            __syncthreads();
        }
        if (do_chan) {
            for (int i = tid; i < n; i += T)
                if (!(set.tag[i] & BB_DEAD)) set.c[i] = __dmul_rn(set.c[i], channel_factor<NW>(P, key_wide<NW>(set.key(i))));
            __syncthreads();
        }
        full = do_chan;
        // ---- commit (every thread keeps the live count and the capacity; thread 0 the totals)
        const int total = n_in + s_cnt[k3][1];
        if (pref && np > acap) acap = max(2 * acap, np);
        if (tid == 0) {
            const int a = s_cnt[k3][2];
            if (B.rec) {
                long long *r = B.rec + 4 * rot;
                r[0] = a;
                r[1] = (pref ? n_in : 0) + np + a;
                r[2] = (pref ? np : 0) + total;
                r[3] = pref ? 1 : 0;
            }
            created += a;
            merge_out += total;
            live_in += n_in;
            peak = max(peak, total);
            early += pref ? 1 : 0;
        }
        alive = total;
        ++rot;
        if (rot >= rot_end || alive > C) break;
    }
    __syncthreads();
    if (s_full && tid == 0) atomicOr(&S->err, ERR_BOUNDS);       // n + alive <= SLOTS: never
    // ---- an index array of the live slots (in the key index's memory)
    unsigned short *sa = reinterpret_cast<unsigned short *>(set.tab);
    {
        int m = 0;
        for (int base = 0; base < n; base += T) {
            const int i = base + tid;
            const int on = i < n && !(set.tag[i] & BB_DEAD) ? 1 : 0;
            int tot;
            const int o = m + block_excl_scan<T>(on, 0, OpSum(), s_scan, &tot);
            if (on) sa[o] = (unsigned short)i;
            m += tot;
        }
        n = m;
    }
    __syncthreads();
    // ---- sort the survivors once (bitonic over an index array; keys are distinct;
    // entries from n up, 0xffff, stay behind every slot)
    int pa = 1;
    while (pa < n) pa <<= 1;
    for (int j = n + tid; j < pa; j += T) sa[j] = 0xffffu;
    __syncthreads();
    for (int k = 2; k <= pa; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int e = tid; e < pa / 2; e += T) {
                const int i = ((e & ~(j - 1)) << 1) | (e & (j - 1)), l = i | j;
                const int u = sa[i], v = sa[l];
                // element u after element v (no order among the entries behind every slot)
                const bool up = (i & k) == 0;
                bool swap;
                if (u == 0xffff || v == 0xffff) swap = u != v && (u == 0xffff) == up;
                else swap = key_lt<NW>(key_wide<NW>(set.key(v)), key_wide<NW>(set.key(u))) == up;
                if (swap) { sa[i] = (unsigned short)v; sa[l] = (unsigned short)u; }
            }
            // pairs less than 32 apart stay within the 64 entries of a warp's 32 threads
            if (j > 32) __syncthreads();
            else __syncwarp();
        }
        __syncthreads();
    }
    // ---- the survivors, dense and sorted, into the other buffer set; <ket|O|ket>
    // of a measured last rotation over the sorted set (contiguous runs per thread,
    // compensated, then lanes and warps in a fixed order)
    u64 *Z = B.z[cur ^ 1], *X = B.x[cur ^ 1];
    double *Cc = B.c[cur ^ 1];
    if ((long long)n > B.cap) {
        if (tid == 0) atomicOr(&S->err, ERR_BOUNDS);
        return;
    }
    const int per = (n + T - 1) / T;
    const int i0 = min(tid * per, n), i1 = min(i0 + per, n);
    Neu acc{0.0, 0.0};
    for (int i = i0; i < i1; ++i) {
        const int src = sa[i];
        const Key<NW> k = key_wide<NW>(set.key(src));
        const double c = set.c[src];
        store_key<NW>(Z, X, i, k);
        Cc[i] = c;
        if (measure_last && is_diag<NW>(k)) acc.add(ket_sign<NW>(k, ket) * c);
    }
    double expect = 0.0;
    if (measure_last) {
        double v = acc.s + acc.c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const double y = __shfl_down_sync(0xffffffffu, v, d);
            if ((lane & (2 * d - 1)) == 0) v += y;
        }
        if (lane == 0) s_red[warp] = v;
        __syncthreads();
        Neu f{0.0, 0.0};
        for (int w = 0; w < T / 32; ++w) f.add(s_red[w]);
        expect = f.s + f.c;
    }
    if (tid == 0) {
        S->n = n;
        S->cur = cur ^ 1;
        S->seg_dense = 1;
        S->rot = rot;
        S->acap_logical = acap;
        S->created += created;
        S->merge_in += live_in + created;
        S->merge_out += merge_out;
        S->live_in += live_in;
        S->early += early;
        S->peak = max(S->peak, (long long)peak);
        S->npref = 0;
        if (measure_last) { S->expect_val = expect; S->measure_valid = 1; }
    }
}

}  // namespace pp
