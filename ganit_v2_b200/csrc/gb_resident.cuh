// On-chip PDHG iterations of small instances: one thread-block cluster keeps
// an instance's scaled matrix, vectors and iterate in shared memory and runs
// a whole check period (check_every iterations) in one launch.
//
// The streaming kernels (gb_pdhg.cuh) pay two dependent launches and a pass
// over the matrix in L2 / HBM per iteration: 7-9 us an iteration on any LP
// below ~1M nonzeros (launch latency), and the L1TEX wavefronts of random
// global gathers on a large batch.  An instance of up to ~100K nonzeros fits
// the shared memory of at most 16 SMs, so here
//   * every CTA of the cluster owns a share of A^T's rows (columns of the LP)
//     and of A's rows, with their matrix entries in shared memory;
//   * every CTA holds a full copy of the two gathered vectors (xbar and y), so
//     a gather is a shared-memory read.  After each half iteration a CTA sends
//     its share to every other one with a bulk copy between shared memories,
//     which counts its bytes on the receiver's mbarrier; the receiver starts
//     its next half when all shares are in.  A CTA that owns nothing on a side
//     (few rows, many columns) sends 16 bytes that nobody reads.  So a share of
//     iteration k + 1 cannot overtake one of iteration k: it depends on the
//     receiver's own share of the half in between, sent after its last read and
//     after all of its shares of iteration k were in.
//
// Layout ("slices").  Rows are reduced by groups of G = 2^lg lanes, lane g of
// a group adding entries g, g + G, ... of its row in order, then the groups'
// shuffle tree -- for FP32 vectors exactly spmv_run's order with the row
// block's own lg, so an FP32 iterate has the same bits on either path.  (FP64
// kernels stream with the segmented order of spmv_run_seg; here lg comes from
// the row's length, and a lane takes its entries as their positions' banks
// allow, which follow the cluster's size: FP64 iterates of an instance may
// differ in their last bits between batches.  Its norm and FP32 iterates do
// not.)  A slice is 32 >> lg rows, one warp; rows are sorted by
// their number of lane steps, so slices carry almost no padding, and a
// slice's entries are stored step-major in pairs: for pair t, 32 words of two
// 16-bit column positions and 32 pairs of values -- conflict-free reads
// whatever the row lengths.  Columns and rows are renumbered by their place
// in that order (owner-major), so an owner's entries are contiguous in the
// gathered vectors.  Padding entries point at a slot that holds 0 with value
// 0; a sum that started at +0 is unchanged by adding +0.
#pragma once
#include <algorithm>
#include <array>
#include <cstring>
#include <vector>

#include "gb_pdhg.cuh"

namespace gb {

constexpr int kResMaxSteps = 32;                       // lane steps of a row (kMaxLaneSum of a STREAM block)
constexpr int kResBins = kResMaxSteps / 2 + 1;         // step pairs 0..16
constexpr int kResMaxIndex = 65535;                    // positions are 16 bits wide
constexpr size_t kResMaxSmem = 227 * 1024;             // shared memory of one CTA
constexpr size_t kResHalfSmem = 113 * 1024;           // of two CTAs on an SM (1 KB each is reserved)
constexpr int kResMaxCluster = 16;
constexpr int kResLaneSteps64 = 8;                     // FP64: lanes per row so that a lane adds at most this many

// One CTA's share of an instance.
struct ResCta {
    int inst;
    int slice0, ns_t, ns_a;   // its slices: ns_t of A^T, then ns_a of A
    int pairs;                // step pairs stored (A^T's slices, then A's)
    int own_t, own_a;         // columns / rows it owns
    int pos_t0, pos_a0;       // their first positions in the instance (multiples of 4: 16-byte copies)
    int n, m;                 // positions of the instance's columns / rows; entries n and m are the zero slots
    int at_t0, at_a0;         // the instance's first entries of col_at / row_at
    int pairs_t;              // A^T's step pairs, stored before A's
    int idle_t, idle_a;       // CTAs of the cluster that own no columns / no rows
    long long pair0;          // first step pair in the packed arrays
};

// A slice in shared memory: {first pair, pairs | lg << 8 | rows << 12, first own index, first position}.
struct ResSlice {
    int pair0, meta, own0, pos0;
};
static_assert(sizeof(ResSlice) == 16, "slices are read as one 16-byte word");

// Launch class: instances with the same cluster size and shared-memory bucket.
struct ResClass {
    int cluster = 1, threads = 256;
    int cta0 = 0, nctas = 0;
    size_t smem = 0;
};

constexpr size_t kResBarBytes = 32;  // two mbarriers, and the 16 bytes of a CTA without a share
constexpr unsigned kResIdleBytes = 16;

// Bytes of a share of `own` entries in the exchange, and of all shares of a
// vector of n positions of which `idle` CTAs own none.
template <class V>
__host__ __device__ inline unsigned share_bytes(int own) {
    return own ? static_cast<unsigned>(sizeof(V)) * ((own + 3) & ~3) : kResIdleBytes;
}
template <class V>
__host__ __device__ inline unsigned share_total(int n, int idle) {
    return static_cast<unsigned>(sizeof(V)) * n + kResIdleBytes * idle;
}

template <class V>
__host__ __device__ inline size_t res_vec_bytes(int n, int m, int own_t, int own_a) {
    auto r4 = [](int k) { return static_cast<size_t>((k + 3) & ~3); };
    return kResBarBytes + sizeof(V) * (r4(n + 1) + r4(m + 1) + 5 * r4(own_t) + 3 * r4(own_a));
}
template <class M, class V>
__host__ __device__ inline size_t res_smem_bytes(int slices, int pairs, int n, int m, int own_t, int own_a) {
    return 16 * static_cast<size_t>(slices) + static_cast<size_t>(pairs) * (128 + 64 * sizeof(M)) +
           res_vec_bytes<V>(n, m, own_t, own_a);
}

// ---------------------------------------------------------------- device
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Barrier over the cluster's threads; what they wrote to any of its shared
// memories before it is visible after it.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_addr(const void* p, int rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(r)
                 : "r"(static_cast<unsigned>(__cvta_generic_to_shared(p))), "r"(rank));
    return r;
}

// mbarriers of one arrival (the CTA's own) plus the bytes announced with it.
__device__ __forceinline__ void mbar_init(unsigned long long* b) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(static_cast<unsigned>(__cvta_generic_to_shared(b)))
                 : "memory");
}
__device__ __forceinline__ void mbar_init_visible() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect(unsigned long long* b, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                     static_cast<unsigned>(__cvta_generic_to_shared(b))),
                 "r"(bytes)
                 : "memory");
}
// Waits for the phase of the given parity; false after kResWaitTries tries
// (each suspends the thread for a while), which only a broken copy can cause.
constexpr int kResWaitTries = 1 << 18;
__device__ __forceinline__ bool mbar_wait(unsigned long long* b, unsigned parity) {
    const unsigned a = static_cast<unsigned>(__cvta_generic_to_shared(b));
    for (int k = 0; k < kResWaitTries; ++k) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// Own shared memory -> the same place of CTA `rank`, counted on its mbarrier.
__device__ __forceinline__ void copy_to_peer(const void* p, unsigned bytes, unsigned long long* bar, int rank) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     cluster_addr(p, rank)),
                 "r"(static_cast<unsigned>(__cvta_generic_to_shared(p))), "r"(bytes), "r"(cluster_addr(bar, rank))
                 : "memory");
}
// Shared-memory writes of this thread, before a bulk copy reads them.
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// End of a half iteration: this CTA's share `p` of a gathered vector goes to
// every other CTA of the cluster, and theirs are awaited (`total`: all shares'
// bytes; `bar`: its mbarrier, at the phase of `parity`).  Returns `lost`, or
// whether the wait ran out; once lost, later waits are skipped.
__device__ __forceinline__ bool cluster_exchange(const void* p, unsigned bytes, unsigned total, unsigned long long* bar,
                                                 unsigned parity, int cluster, int rank, bool lost) {
    if (cluster == 1) {
        __syncthreads();
        return lost;
    }
    fence_async_proxy();
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        if (lane == 0) mbar_expect(bar, total - bytes);
        if (lane < cluster && lane != rank) copy_to_peer(p, bytes, bar, lane);
    }
    return lost || !mbar_wait(bar, parity);
}

// End of a CTA's work: it does not leave while a copy may still read its share.
// Copies to it are in, since it awaited them, unless a wait ran out: then it
// stays for about a millisecond after every CTA has sent its last (a copy takes
// microseconds).
__device__ __forceinline__ void cluster_leave(int cluster, bool lost) {
    if (cluster == 1) return;
    cluster_sync();
    if (lost)
        for (int k = 0; k < 64; ++k) __nanosleep(16000);
}

// Two matrix values of a lane's step pair.
__device__ __forceinline__ void ld_pair(const float* p, float& a, float& b) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    a = v.x; b = v.y;
}
__device__ __forceinline__ void ld_pair(const double* p, double& a, double& b) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    a = v.x; b = v.y;
}
__device__ __forceinline__ void ld_pair(const __nv_bfloat16* p, __nv_bfloat16& a, __nv_bfloat16& b) {
    const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(p);
    a = v.x; b = v.y;
}

// Sum over the group of 2^lg lanes, into its first lane (reduce_rows' tree).
template <class V>
__device__ __forceinline__ V group_tree(V acc, int lg) {
    if (lg > 4) acc += __shfl_down_sync(0xffffffffu, acc, 16);
    if (lg > 3) acc += __shfl_down_sync(0xffffffffu, acc, 8);
    if (lg > 2) acc += __shfl_down_sync(0xffffffffu, acc, 4);
    if (lg > 1) acc += __shfl_down_sync(0xffffffffu, acc, 2);
    if (lg > 0) acc += __shfl_down_sync(0xffffffffu, acc, 1);
    return acc;
}

// Row sums of a slice: a lane's part over its steps, then the group's tree
// (the sum lands in each group's first lane).
template <class M, class V>
__device__ __forceinline__ V slice_sum(int pair0, int np, int lg, const unsigned* idx, const M* val, const V* g,
                                       int lane) {
    const unsigned* ip = idx + pair0 * 32 + lane;
    const M* vp = val + pair0 * 64 + 2 * lane;
    V acc = V(0);
#pragma unroll 4
    for (int t = 0; t < np; ++t) {
        const unsigned j = ip[32 * t];
        M a, b;
        ld_pair(vp + 64 * t, a, b);
        acc += static_cast<V>(a) * g[j & 0xffffu];
        acc += static_cast<V>(b) * g[j >> 16];
    }
    return group_tree(acc, lg);
}

// A slice of up to kResRegPairs pairs held in registers across a launch: its
// sums read shared memory for the gathers alone (a pair's positions and values
// are 3 of its ~10.7 wavefronts in FP32, 5 of ~18 in FP64).  Pairs past the end
// are padding (the zero slot with value 0).  For CTAs of 256 threads: LP
// 701 x 1753 3.74 -> 3.25 ms; with 512 threads it costs the second CTA per SM
// (37 LPs 2.86 -> 3.3 ms) and gains nothing where the exchange is the longer
// part (LP 2000 x 5000).
constexpr int kResRegPairs = 8;
template <class M>
struct RegSlice {
    unsigned j[kResRegPairs];
    M v[2 * kResRegPairs];
    __device__ __forceinline__ void load(const ResSlice& e, const unsigned* idx, const M* val, unsigned zero, int lane) {
        const int np = e.meta & 0xff;
#pragma unroll
        for (int t = 0; t < kResRegPairs; ++t) {
            j[t] = zero;
            v[2 * t] = v[2 * t + 1] = static_cast<M>(0.0f);
            if (t < np) {
                j[t] = idx[(e.pair0 + t) * 32 + lane];
                ld_pair(val + (e.pair0 + t) * 64 + 2 * lane, v[2 * t], v[2 * t + 1]);
            }
        }
    }
    template <class V>
    __device__ __forceinline__ V sum(int np, int lg, const V* g) const {
        V acc = V(0);
#pragma unroll
        for (int h = 0; h < kResRegPairs; h += 4) {
            if (h < np) {
                V x[8];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    x[2 * t] = g[j[h + t] & 0xffffu];
                    x[2 * t + 1] = g[j[h + t] >> 16];
                }
#pragma unroll
                for (int t = 0; t < 8; ++t) acc += static_cast<V>(v[2 * h + t]) * x[t];
            }
        }
        return group_tree(acc, lg);
    }
};

template <class M, class V>
struct ResArgs {
    const ResCta* cta;        // records of this class
    const ResSlice* slices;
    const unsigned* idx;      // packed position pairs
    const M* val;             // packed value pairs
    const int* col_at;        // position -> column (global), per instance from its first column
    const int* row_at;
    const V* x0; const V* y0; // iterate in
    V* x; V* y;               // iterate out
    V* sumx; V* sumy;
    const V* c; const V* l; const V* u; const V* lo; const V* hi;
    SolveState* st;
    int* error;               // set when a wait ran out
    int iters, cluster;
};

template <class M, class V, int T>
__global__ void __launch_bounds__(T, T < 1024 ? 2 : 1) k_resident(const __grid_constant__ ResArgs<M, V> a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const ResCta r = a.cta[blockIdx.x];
    const SolveState& s = a.st[r.inst];
    if (s.active == 0) return;  // the same for every CTA of the cluster
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int W = T / 32;
    auto r4 = [](int k) { return (k + 3) & ~3; };
    // the gathered vectors first: their place is the same in every CTA of the cluster
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem);  // [0] xbar, [1] y
    V* xs = reinterpret_cast<V*>(smem + kResBarBytes);  // xbar by position, all columns
    V* ys = xs + r4(r.n + 1);                          // y by position, all rows
    ResSlice* sl = reinterpret_cast<ResSlice*>(ys + r4(r.m + 1));
    unsigned* idx = reinterpret_cast<unsigned*>(sl + r.ns_t + r.ns_a);
    M* val = reinterpret_cast<M*>(idx + 32 * r.pairs);
    V* ox = reinterpret_cast<V*>(val + 64 * r.pairs);
    V* oc = ox + r4(r.own_t);
    V* ol = oc + r4(r.own_t);
    V* ou = ol + r4(r.own_t);
    V* osx = ou + r4(r.own_t);
    V* olo = osx + r4(r.own_t);
    V* ohi = olo + r4(r.own_a);
    V* osy = ohi + r4(r.own_a);
    // matrix share and slice table: asynchronous copies; vectors meanwhile
    for (int k = tid; k < r.ns_t + r.ns_a; k += T) cp_async16(sl + k, a.slices + r.slice0 + k);
    for (int k = tid; k < 8 * r.pairs; k += T) cp_async16(idx + 4 * k, a.idx + 32 * r.pair0 + 4 * k);
    constexpr int kPer16 = 16 / static_cast<int>(sizeof(M));
    for (int k = tid; k < 64 / kPer16 * r.pairs; k += T) cp_async16(val + kPer16 * k, a.val + 64 * r.pair0 + kPer16 * k);
    for (int k = tid; k < r.own_t; k += T) {
        const int j = a.col_at[r.at_t0 + r.pos_t0 + k];
        ox[k] = a.x0[j];
        oc[k] = a.c[j];
        ol[k] = a.l[j];
        ou[k] = a.u[j];
        osx[k] = a.sumx[j];
    }
    for (int k = tid; k < r.own_a; k += T) {
        const int i = a.row_at[r.at_a0 + r.pos_a0 + k];
        olo[k] = a.lo[i];
        ohi[k] = a.hi[i];
        osy[k] = a.sumy[i];
    }
    for (int k = tid; k < r.m; k += T) {
        const int i = a.row_at[r.at_a0 + k];
        ys[k] = i >= 0 ? a.y0[i] : V(0);  // -1: between two shares
    }
    if (tid == 0) {
        xs[r.n] = V(0);
        ys[r.m] = V(0);
        mbar_init(bar);
        mbar_init(bar + 1);
        mbar_init_visible();
    }
    const V tau = static_cast<V>(s.tau), sigma = static_cast<V>(s.sigma);
    cp_async_wait_all();
    const int rank = static_cast<int>(blockIdx.x) % a.cluster;
    const unsigned bytes_x = share_bytes<V>(r.own_t), bytes_y = share_bytes<V>(r.own_a);
    const unsigned total_x = share_total<V>(r.n, r.idle_t), total_y = share_total<V>(r.m, r.idle_a);
    const void* const idle = smem + kResBarBytes - kResIdleBytes;
    const void* const mine_x = r.own_t ? xs + r.pos_t0 : idle;
    const void* const mine_y = r.own_a ? ys + r.pos_a0 : idle;
    bool lost = false;
    auto exchange = [&](const void* p, unsigned bytes, unsigned total, int b, int it) {
        lost = cluster_exchange(p, bytes, total, bar + b, it & 1, a.cluster, rank, lost);
    };
    if (a.cluster > 1) cluster_sync();  // every CTA has started and holds its share
    else __syncthreads();
    // each warp's first slice of either side in registers
    RegSlice<M> reg_t, reg_a;
    bool has_t = false, has_a = false;
    constexpr bool kReg = T <= 256;  // larger CTAs keep 64 registers a thread, so that two share an SM
    if (kReg && warp < r.ns_t) {
        const ResSlice e = sl[warp];
        has_t = (e.meta & 0xff) <= kResRegPairs;
        if (has_t) reg_t.load(e, idx, val, static_cast<unsigned>(r.m) * 0x10001u, lane);
    }
    if (kReg && warp < r.ns_a) {
        const ResSlice e = sl[r.ns_t + warp];
        has_a = (e.meta & 0xff) <= kResRegPairs;
        if (has_a) reg_a.load(e, idx, val, static_cast<unsigned>(r.n) * 0x10001u, lane);
    }
    for (int it = 0; it < a.iters; ++it) {
        for (int q = warp; q < r.ns_t; q += W) {  // primal half (PrimalEpi)
            const ResSlice e = sl[q];
            const int np = e.meta & 0xff, lg = (e.meta >> 8) & 0xf, nr = e.meta >> 12, grp = min(lane >> lg, nr - 1);
            const int k = e.own0 + grp;
            const V xk = ox[k], ck = oc[k], lk = ol[k], uk = ou[k], sk = osx[k];
            const V t = kReg && q == warp && has_t ? reg_t.template sum<V>(np, lg, ys)
                                           : slice_sum<M, V>(e.pair0, np, lg, idx, val, ys, lane);
            const V g = ck - t + V(0);
            V v = xk - tau * g;
            v = (v < lk) ? lk : v;
            v = (uk < v) ? uk : v;
            if ((lane & ((1 << lg) - 1)) == 0 && (lane >> lg) < nr) {
                ox[k] = v;
                osx[k] = sk + v;
                xs[e.pos0 + grp] = V(2) * v - xk;
            }
        }
        exchange(mine_x, bytes_x, total_x, 0, it);
        for (int q = r.ns_t + warp; q < r.ns_t + r.ns_a; q += W) {  // dual half (DualEpi)
            const ResSlice e = sl[q];
            const int np = e.meta & 0xff, lg = (e.meta >> 8) & 0xf, nr = e.meta >> 12, grp = min(lane >> lg, nr - 1);
            const int k = e.own0 + grp;
            const V yk = ys[e.pos0 + grp], sk = osy[k], lk = sigma * olo[k], hk = sigma * ohi[k];
            const V t = kReg && q == r.ns_t + warp && has_a ? reg_a.template sum<V>(np, lg, xs)
                                                    : slice_sum<M, V>(e.pair0, np, lg, idx, val, xs, lane);
            const V qv = yk - sigma * t;
            V w = -qv;
            w = (w < lk) ? lk : w;
            w = (hk < w) ? hk : w;
            const V v = qv + w;
            if ((lane & ((1 << lg) - 1)) == 0 && (lane >> lg) < nr) {
                osy[k] = sk + v;
                ys[e.pos0 + grp] = v;
            }
        }
        exchange(mine_y, bytes_y, total_y, 1, it);
    }
    if (lost) {  // the solve stops at the coming check and reports the error
        atomicExch(a.error, 1);
        a.st[r.inst].max_iter = 0;
    }
    for (int k = tid; k < r.own_t; k += T) {
        const int j = a.col_at[r.at_t0 + r.pos_t0 + k];
        a.x[j] = ox[k];
        a.sumx[j] = osx[k];
    }
    for (int k = tid; k < r.own_a; k += T) {
        const int i = a.row_at[r.at_a0 + r.pos_a0 + k];
        a.y[i] = ys[r.pos_a0 + k];
        a.sumy[i] = osy[k];
    }
    cluster_leave(a.cluster, lost);
}

// Power iteration on A'^T A' (scaling.cpp:131-155) of the resident instances on
// the FP64 plan: 50 steps in one launch instead of 200 launches (0.6 - 1 ms of
// a small LP's set-up; 0.1 - 0.2 ms here).  z is in xs and w in ys; after z's
// exchange every CTA forms ||z|| over all of it, in the order of the columns
// (k_seg_red's), not of their positions: the norm, and with it the step sizes,
// must not depend on the cluster's size, which follows what shares the batch.
inline size_t power_smem_bytes(const ResCta& c) {
    return res_smem_bytes<double, double>(c.ns_t + c.ns_a, c.pairs, c.n, c.m, 0, 0) + 8 * 32;
}
struct PowerArgs {
    const ResCta* cta;
    const ResSlice* slices;
    const unsigned* idx;
    const double* val;
    const unsigned short* pos_t;  // column -> position
    const int* col_off;           // instance -> first column
    double* scal;          // per instance rows of kScal; [lambda] is written
    int scal_stride, lambda;
    int* error;
    int iters, cluster;
};
template <int T>
__global__ void __launch_bounds__(T, T < 1024 ? 2 : 1) k_power_chip(const __grid_constant__ PowerArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const ResCta r = a.cta[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int W = T / 32;
    auto r4 = [](int k) { return (k + 3) & ~3; };
    unsigned long long* bar = reinterpret_cast<unsigned long long*>(smem);
    double* xs = reinterpret_cast<double*>(smem + kResBarBytes);
    double* ys = xs + r4(r.n + 1);
    ResSlice* sl = reinterpret_cast<ResSlice*>(ys + r4(r.m + 1));
    unsigned* idx = reinterpret_cast<unsigned*>(sl + r.ns_t + r.ns_a);
    double* val = reinterpret_cast<double*>(idx + 32 * r.pairs);
    double* red = val + 64 * r.pairs;
    for (int k = tid; k < r.ns_t + r.ns_a; k += T) cp_async16(sl + k, a.slices + r.slice0 + k);
    for (int k = tid; k < 8 * r.pairs; k += T) cp_async16(idx + 4 * k, a.idx + 32 * r.pair0 + 4 * k);
    for (int k = tid; k < 32 * r.pairs; k += T) cp_async16(val + 2 * k, a.val + 64 * r.pair0 + 2 * k);
    if (tid == 0) {
        xs[r.n] = 0.0;
        ys[r.m] = 0.0;
        mbar_init(bar);
        mbar_init(bar + 1);
        mbar_init_visible();
    }
    const int rank = static_cast<int>(blockIdx.x) % a.cluster;
    const unsigned bytes_x = share_bytes<double>(r.own_t), bytes_y = share_bytes<double>(r.own_a);
    const unsigned total_x = share_total<double>(r.n, r.idle_t), total_y = share_total<double>(r.m, r.idle_a);
    const void* const idle = smem + kResBarBytes - kResIdleBytes;
    const void* const mine_x = r.own_t ? xs + r.pos_t0 : idle;
    const void* const mine_y = r.own_a ? ys + r.pos_a0 : idle;
    const int c0 = a.col_off[r.inst], c1 = a.col_off[r.inst + 1];
    cp_async_wait_all();
    if (a.cluster > 1) cluster_sync();
    else __syncthreads();
    for (int k = tid; k < r.own_t; k += T) xs[r.pos_t0 + k] = 1.0;  // v = 1 / ||1||: the first ||z|| is sqrt(n)
    bool lost = false;
    double lambda = 0.0;
    for (int it = 0; it <= a.iters; ++it) {
        lost = cluster_exchange(mine_x, bytes_x, total_x, bar, it & 1, a.cluster, rank, lost);
        double s = 0.0;
        if (warp < kWarps) {
#pragma unroll 4
            for (int j = c0 + tid; j < c1; j += kThreads) {
                const double z = xs[a.pos_t[j]];
                s += z * z;
            }
            s = warp_sum(s);
            if (lane == 0) red[warp] = s;
        }
        __syncthreads();
        double nz = 0.0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) nz += red[w];
        nz = sqrt(nz);
        if (it > 0 && nz != 0.0) lambda = nz;
        if (it == a.iters || nz == 0.0) break;  // the same in every CTA
        // w = A z / ||z||: z itself stays as it is while peers may still copy it
        for (int q = r.ns_t + warp; q < r.ns_t + r.ns_a; q += W) {
            const ResSlice e = sl[q];
            const int lg = (e.meta >> 8) & 0xf;
            const double t = slice_sum<double, double>(e.pair0, e.meta & 0xff, lg, idx, val, xs, lane);
            if ((lane & ((1 << lg) - 1)) == 0 && (lane >> lg) < (e.meta >> 12)) ys[e.pos0 + (lane >> lg)] = t / nz;
        }
        lost = cluster_exchange(mine_y, bytes_y, total_y, bar + 1, it & 1, a.cluster, rank, lost);
        for (int q = warp; q < r.ns_t; q += W) {
            const ResSlice e = sl[q];
            const int lg = (e.meta >> 8) & 0xf;
            const double t = slice_sum<double, double>(e.pair0, e.meta & 0xff, lg, idx, val, ys, lane);
            if ((lane & ((1 << lg) - 1)) == 0 && (lane >> lg) < (e.meta >> 12)) xs[e.pos0 + (lane >> lg)] = t;
        }
    }
    if (lost && tid == 0) atomicExch(a.error, 1);
    if (rank == 0 && tid == 0) a.scal[static_cast<size_t>(r.inst) * a.scal_stride + a.lambda] = lambda;
    cluster_leave(a.cluster, lost);
}

// ---------------------------------------------------------------- packing (device, once per plan)
// Lanes per row: lg of the STREAM block that holds it (FP32 vectors).
static __global__ void k_res_row_lg(int nb, const RowBlock* __restrict__ blocks, unsigned char* __restrict__ lg) {
    const RowBlock b = blocks[blockIdx.x];
    for (int r = b.r0 + threadIdx.x; r < b.r1; r += blockDim.x) lg[r] = static_cast<unsigned char>(b.lg);
}
__host__ __device__ inline int res_lg64(int len) {
    int lg = 0;
    while (lg < 5 && (kResLaneSteps64 << lg) < len) ++lg;
    return lg;
}

// One side (A^T's or A's rows) of one resident instance, for the packing kernels.
struct ResSide {
    int row0, row1;                        // global rows of the side's matrix
    int at0;                               // first entry of the position -> row list
    int slice0[6];                         // first entry of the side's slices of each lg in the slice list
    int rank0[6][kResBins];                // rank of the first row of (lg, pairs) among the rows of lg
};
struct ResSliceAt {                        // slice list entry: where the slice lives
    long long pair0;                       // global first pair
    int meta, pos0;
    int at0, side;                         // its instance's first entry of the side's position -> row list; 0: A^T
    int zero;                              // the gathered vector's zero slot
};

// One warp per side walks its rows in order and gives every row its slot
// (slice list entry * 32 + group) and its position.
static __global__ void k_res_rank(const ResSide* __restrict__ sides, const int* __restrict__ ptr,
                                  const unsigned char* __restrict__ lg_of, const ResSliceAt* __restrict__ slices,
                                  int* __restrict__ slot, unsigned short* __restrict__ pos, int* __restrict__ at) {
    __shared__ int next[6 * kResBins];
    const ResSide& sd = sides[blockIdx.x];
    const int lane = threadIdx.x;
    for (int k = lane; k < 6 * kResBins; k += 32) next[k] = sd.rank0[k / kResBins][k % kResBins];
    __syncwarp();
    for (int r0 = sd.row0; r0 < sd.row1; r0 += 32) {
        const int r = r0 + lane;
        int bin = -1, lg = 0;
        if (r < sd.row1) {
            const int len = ptr[r + 1] - ptr[r];
            lg = lg_of ? lg_of[r] : res_lg64(len);
            const int steps = (len + (1 << lg) - 1) >> lg;
            bin = lg * kResBins + ((steps + 1) >> 1);
        }
        const unsigned peers = __match_any_sync(0xffffffffu, bin);
        const int rank = __popc(peers & ((1u << lane) - 1u));
        int base = 0;
        if (bin >= 0) base = next[bin];
        __syncwarp();
        if (bin >= 0 && rank == 0) next[bin] = base + __popc(peers);
        __syncwarp();
        if (bin >= 0) {
            const int k = base + rank, rows = 32 >> lg;
            const int e = sd.slice0[lg] + k / rows, grp = k % rows;
            const int p = slices[e].pos0 + grp;
            slot[r] = e * 32 + grp;
            if (pos) pos[r] = static_cast<unsigned short>(p);
            at[sd.at0 + p] = r;
        }
    }
}

// Every packed pair starts as padding: the zero slot's position, value 0.
static __global__ void k_res_fill(const ResCta* __restrict__ cta, unsigned* __restrict__ idx) {
    const ResCta r = cta[blockIdx.x];
    // A^T's pairs gather y (zero slot m), A's gather xbar (zero slot n)
    const unsigned zt = static_cast<unsigned>(r.m) * 0x10001u, za = static_cast<unsigned>(r.n) * 0x10001u;
    for (int k = threadIdx.x; k < 32 * r.pairs; k += blockDim.x) idx[32 * r.pair0 + k] = k < 32 * r.pairs_t ? zt : za;
}

// FP64: the step of every entry, chosen so that the 16 lanes of a half warp
// gather from as many different pairs of banks as can be had (the order of a
// lane's sum is free there; random positions take 3.1 wavefronts a half, these
// ~2).  One warp per slice: lane by lane, both halves side by side, each entry
// goes to the free step whose bank pair is least used so far, with its position
// and (`val` given) its value.  Positions, and so the order of the sums, follow
// the cluster's size, which follows what shares the batch; the power iteration
// therefore runs before, on entries in the matrix's order.  Measured, FP64:
// LP 2000 x 5000 2.25 -> 2.18 ms, 37 LPs 2.86 -> 2.76, 64 branching children
// 161 -> 155.
struct ResOrderSide {
    const int *at, *ptr, *col;          // position -> row, the rows
    const double* val;
    const unsigned short* pos_other;    // positions of the gathered vector
    unsigned char* step;
};
struct ResOrderArgs {
    ResOrderSide side[2];
    unsigned short* idx;
    double* val;                        // packed values, or nullptr: positions alone
};
static __global__ void __launch_bounds__(128) k_res_order(int nslices, const ResSliceAt* __restrict__ slices,
                                                          const __grid_constant__ ResOrderArgs a) {
    __shared__ unsigned char load[4][2][kResMaxSteps][16];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, half = lane >> 4;
    for (int z = lane; z < 2 * kResMaxSteps * 16; z += 32) (&load[w][0][0][0])[z] = 0;
    __syncwarp();
    const int q = blockIdx.x * 4 + w;
    if (q >= nslices) return;
    const ResSliceAt e = slices[q];
    const ResOrderSide& d = a.side[e.side];
    const int steps = 2 * (e.meta & 0xff), lg = (e.meta >> 8) & 0xf, nr = e.meta >> 12, G = 1 << lg, grp = lane >> lg;
    int p0 = 0, len = 0;
    if (grp < nr) {
        const int r = d.at[e.at0 + e.pos0 + grp];
        p0 = d.ptr[r];
        len = d.ptr[r + 1] - p0;
    }
    auto put = [&](int t, int pos, double v) {
        const long long z = (e.pair0 + (t >> 1)) * 64 + 2 * lane + (t & 1);
        a.idx[z] = static_cast<unsigned short>(pos);
        if (a.val) a.val[z] = v;
    };
    unsigned taken = 0u;
    for (int l = 0; l < 16; ++l) {
        if ((lane & 15) == l) {
            for (int k = lane & (G - 1); k < len; k += G) {
                const int pos = d.pos_other[d.col[p0 + k]], bank = pos & 15;
                int best = 0, least = 255;
                for (int t = 0; t < steps; ++t) {
                    const int u = load[w][half][t][bank];
                    if (!(taken >> t & 1u) && u < least) {
                        least = u;
                        best = t;
                    }
                }
                taken |= 1u << best;
                ++load[w][half][best][bank];
                d.step[p0 + k] = static_cast<unsigned char>(best);
                put(best, pos, a.val ? d.val[p0 + k] : 0.0);
            }
        }
        __syncwarp();
    }
    for (int t = 0; t < steps; ++t)
        if (!(taken >> t & 1u)) put(t, e.zero, 0.0);
}

// Entries of the rows of one side: positions (from the other side's
// numbering) and, through k_res_values, values.
static __global__ void k_res_entries(int rows, const int* __restrict__ ptr, const int* __restrict__ col,
                                     const int* __restrict__ slot, const ResSliceAt* __restrict__ slices,
                                     const unsigned short* __restrict__ pos_other,
                                     unsigned short* __restrict__ idx) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        const int sr = slot[r];
        if (sr < 0) continue;  // the row's instance is not resident
        const ResSliceAt e = slices[sr >> 5];
        const int lg = (e.meta >> 8) & 0xf, G = 1 << lg, p0 = ptr[r], len = ptr[r + 1] - p0;
        for (int k = 0; k < len; ++k) {
            const int t = k >> lg, lane = ((sr & 31) << lg) + (k & (G - 1));
            idx[(e.pair0 + (t >> 1)) * 64 + 2 * lane + (t & 1)] = pos_other[col[p0 + k]];
        }
    }
}
template <class M, class S>
__global__ void k_res_values(int rows, const int* __restrict__ ptr, const S* __restrict__ val,
                             const int* __restrict__ slot, const ResSliceAt* __restrict__ slices,
                             const unsigned char* __restrict__ step, M* __restrict__ out) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x) {
        const int sr = slot[r];
        if (sr < 0) continue;
        const ResSliceAt e = slices[sr >> 5];
        const int lg = (e.meta >> 8) & 0xf, G = 1 << lg, p0 = ptr[r], len = ptr[r + 1] - p0;
        for (int k = 0; k < len; ++k) {
            const int t = step ? step[p0 + k] : k >> lg, lane = ((sr & 31) << lg) + (k & (G - 1));
            out[(e.pair0 + (t >> 1)) * 64 + 2 * lane + (t & 1)] = static_cast<M>(val[p0 + k]);
        }
    }
}

// ---------------------------------------------------------------- host: who is resident, and where
// Row counts of one side by (lg, step pairs); false: a row it cannot hold.
struct ResHist {
    int h[6][kResBins] = {};
    long long pairs = 0;  // over slices
    int slices = 0;
    // slices of each lg: pairs of the k-th (rows in order of falling pairs)
    template <class F>
    void each_slice(F&& f) const {
        for (int lg = 0; lg < 6; ++lg) {
            const int rows = 32 >> lg;
            int left = 0, fill = 0, top = 0;
            for (int b = kResBins - 1; b >= 0; --b) left += h[lg][b];
            for (int b = kResBins - 1; b >= 0 && left > 0; --b) {
                int c = h[lg][b];
                while (c > 0) {
                    if (fill == 0) top = b;
                    const int take = std::min(c, rows - fill);
                    fill += take;
                    c -= take;
                    left -= take;
                    if (fill == rows || left == 0) {
                        f(lg, top, fill);
                        fill = 0;
                    }
                }
            }
        }
    }
    void count() {
        pairs = 0;
        slices = 0;
        each_slice([&](int, int np, int) {
            pairs += np;
            ++slices;
        });
    }
};
inline bool res_hist_rows(const int* ptr, int r0, int r1, int lg_fixed, ResHist& H) {
    for (int r = r0; r < r1; ++r) {
        const int len = ptr[r + 1] - ptr[r];
        const int lg = lg_fixed >= 0 ? lg_fixed : res_lg64(len);
        const int steps = (len + (1 << lg) - 1) >> lg;
        if (steps > kResMaxSteps) return false;
        ++H.h[lg][(steps + 1) >> 1];
    }
    return true;
}

// Slices of both sides of an instance dealt to C CTAs: by falling pairs, back
// and forth over the CTAs, so the shares differ by about one slice.
struct ResDeal {
    struct Item {
        int lg, pairs, rows, cta, ord;  // ord: place among the CTA's slices of its side
        int own0, pos0, pair0;
    };
    std::vector<Item> side[2];      // A^T, A; in slice list order (lg-major)
    std::vector<ResCta> cta;
    size_t smem(size_t sm, size_t sv) const {
        size_t top = 0;
        for (const ResCta& c : cta) {
            const size_t b = sm == 8 ? res_smem_bytes<double, double>(c.ns_t + c.ns_a, c.pairs, c.n, c.m, c.own_t, c.own_a)
                             : sv == 8 ? res_smem_bytes<float, double>(c.ns_t + c.ns_a, c.pairs, c.n, c.m, c.own_t, c.own_a)
                                       : res_smem_bytes<float, float>(c.ns_t + c.ns_a, c.pairs, c.n, c.m, c.own_t, c.own_a);
            top = std::max(top, b);
        }
        return top;
    }
};
inline void res_deal(const std::array<ResHist, 2>& H, int C, ResDeal& D) {
    D.cta.assign(C, ResCta{});
    for (int sd = 0; sd < 2; ++sd) {
        auto& it = D.side[sd];
        it.clear();
        it.reserve(H[sd].slices);
        H[sd].each_slice([&](int lg, int np, int rows) { it.push_back({lg, np, rows, 0, 0, 0, 0, 0}); });
        std::vector<int> order(it.size());
        std::array<int, kResBins + 1> start{};
        for (const auto& e : it) ++start[kResBins - 1 - e.pairs + 1];
        for (int b = 0; b < kResBins; ++b) start[b + 1] += start[b];
        for (size_t k = 0; k < it.size(); ++k) order[start[kResBins - 1 - it[k].pairs]++] = static_cast<int>(k);
        std::vector<int> own(C, 0);
        for (size_t q = 0; q < order.size(); ++q) {
            const int lap = static_cast<int>(q / C), at = static_cast<int>(q % C);
            const int c = (lap & 1) ? C - 1 - at : at;
            auto& e = it[order[q]];
            ResCta& k = D.cta[c];
            e.cta = c;
            e.ord = sd == 0 ? k.ns_t++ : k.ns_a++;
            e.pair0 = k.pairs;
            e.own0 = own[c];
            own[c] += e.rows;
            k.pairs += e.pairs;
        }
        int pos = 0;
        for (int c = 0; c < C; ++c) {
            (sd == 0 ? D.cta[c].own_t : D.cta[c].own_a) = own[c];
            (sd == 0 ? D.cta[c].pos_t0 : D.cta[c].pos_a0) = pos;
            pos += (own[c] + 3) & ~3;
            if (sd == 0) D.cta[c].pairs_t = D.cta[c].pairs;
        }
        const int idle = static_cast<int>(std::count(own.begin(), own.end(), 0));
        for (ResCta& k : D.cta) {
            (sd == 0 ? k.n : k.m) = pos;
            (sd == 0 ? k.idle_t : k.idle_a) = idle;
        }
        for (auto& e : it) e.pos0 = (sd == 0 ? D.cta[e.cta].pos_t0 : D.cta[e.cta].pos_a0) + e.own0;
    }
}

// Device tables of the resident instances, filled instance by instance.
struct ResTables {
    std::vector<ResCta> cta;
    std::vector<ResSlice> slices;
    std::vector<ResSliceAt> at;
    std::vector<ResSide> sides[2];  // A^T, A
    long long pairs = 0;
    int positions[2] = {0, 0};      // entries of col_at, row_at
    void add(int inst, const std::array<ResHist, 2>& H, const ResDeal& D, int col0, int col1, int row0, int row1) {
        const size_t c0 = cta.size();
        for (ResCta k : D.cta) {
            k.inst = inst;
            k.at_t0 = positions[0];
            k.at_a0 = positions[1];
            k.pair0 = pairs;
            k.slice0 = static_cast<int>(slices.size());
            pairs += k.pairs;
            slices.resize(slices.size() + k.ns_t + k.ns_a);
            cta.push_back(k);
        }
        for (int sd = 0; sd < 2; ++sd) {
            ResSide s{};
            s.row0 = sd == 0 ? col0 : row0;
            s.row1 = sd == 0 ? col1 : row1;
            s.at0 = positions[sd];
            for (int lg = 0; lg < 6; ++lg) {
                int run = 0;
                for (int b = kResBins - 1; b >= 0; --b) {
                    s.rank0[lg][b] = run;
                    run += H[sd].h[lg][b];
                }
                s.slice0[lg] = -1;
            }
            for (const auto& e : D.side[sd]) {
                if (s.slice0[e.lg] < 0) s.slice0[e.lg] = static_cast<int>(at.size());
                const ResCta& k = cta[c0 + e.cta];
                const int meta = e.pairs | e.lg << 8 | e.rows << 12;
                at.push_back({k.pair0 + e.pair0, meta, e.pos0, positions[sd], sd, sd == 0 ? k.m : k.n});
                slices[k.slice0 + (sd == 0 ? 0 : k.ns_t) + e.ord] = {e.pair0, meta, e.own0, e.pos0};
            }
            sides[sd].push_back(s);
        }
        positions[0] += D.cta[0].n;
        positions[1] += D.cta[0].m;
    }
};

// Pinned and device memory that a plan needs only while it is packed.
struct PlanScratch {
    std::vector<void*> pinned;  // sources of the plans' copies
    std::vector<DevBuf<unsigned char>> dev;
    size_t dev_bytes() const {
        size_t b = 0;
        for (const auto& d : dev) b += d.size();
        return b;
    }
    // Gives it back; the stream that packed has to be idle.
    void release() {
        if (pinned.empty() && dev.empty()) return;
        begin_free_batch();
        for (void* p : pinned) host_free(p);
        pinned.clear();
        dev.clear();
        end_free_batch();
    }
};

// Device arrays of a plan in one allocation (a cudaMalloc each took longer
// than packing a small LP), those filled by the host in one copy, those that
// start as -1 in one memset.  The copy's source is pinned, so the host goes on
// while earlier work of the stream runs; it stays in `scratch` until released.
class PlanArena {
   public:
    template <class T>
    void host(T*& p, const std::vector<T>& v) {
        add(reinterpret_cast<void**>(&p), v.size() * sizeof(T), 0, v.data());
    }
    template <class T>
    void ones(T*& p, size_t n) { add(reinterpret_cast<void**>(&p), n * sizeof(T), 1, nullptr); }
    template <class T>
    void raw(T*& p, size_t n) { add(reinterpret_cast<void**>(&p), n * sizeof(T), 2, nullptr); }
    void commit(DevBuf<unsigned char>& mem, PlanScratch& scratch, cudaStream_t s) {
        size_t end[3], off = 0;
        for (int kind = 0; kind < 3; ++kind) {
            for (Item& i : items_)
                if (i.kind == kind) {
                    i.off = off;
                    off += (i.bytes + 255) & ~size_t(255);
                }
            end[kind] = off;
        }
        mem.reset(std::max<size_t>(off, 256));
        unsigned char* stage = nullptr;
        if (end[0]) {
            stage = static_cast<unsigned char*>(host_alloc(end[0]));
            scratch.pinned.push_back(stage);
        }
        for (const Item& i : items_) {
            *i.slot = mem.get() + i.off;
            if (i.kind == 0 && i.bytes) std::memcpy(stage + i.off, i.src, i.bytes);
        }
        mem.upload(stage, end[0], s);
        if (end[1] > end[0]) GB_CUDA(cudaMemsetAsync(mem.get() + end[0], 0xff, end[1] - end[0], s));
    }

   private:
    struct Item {
        void** slot;
        size_t bytes;
        int kind;
        const void* src;
        size_t off;
    };
    std::vector<Item> items_;
    void add(void** slot, size_t bytes, int kind, const void* src) { items_.push_back({slot, bytes, kind, src, 0}); }
};

// The resident instances of a problem for one vector precision.
struct ResPlan {
    bool built = false;
    std::vector<char> resident;             // per instance
    std::vector<ResClass> classes;
    DevBuf<unsigned char> mem;              // everything below but the values
    ResCta* cta = nullptr;
    ResSlice* slices = nullptr;
    ResSliceAt* at = nullptr;
    ResSide *sides_t = nullptr, *sides_a = nullptr;
    unsigned* idx = nullptr;
    int *col_at = nullptr, *row_at = nullptr, *slot_t = nullptr, *slot_a = nullptr;
    unsigned short *pos_t = nullptr, *pos_a = nullptr;
    unsigned char *lg_t = nullptr, *lg_a = nullptr;      // FP32
    unsigned char *step_t = nullptr, *step_a = nullptr;  // FP64: k_res_order
    bool ordered = false;                                // whether the entries lie in that order
    DevBuf<float> val32;
    DevBuf<double> val64;
    DevBuf<__nv_bfloat16> valbf;
    long long pairs = 0;
    int nslices = 0;
    // Row blocks of the other instances, which the streaming kernels run
    // (nothing: every instance is resident), by matrix type (0: FP32 / BF16,
    // 1: FP64): a block's bitmap, slots and counter are those of the schedule
    // it was cut for, and the two types' schedules part when they are tuned.
    RowBlock *list_a[2] = {}, *list_t[2] = {};
    int list_na[2] = {}, list_nt[2] = {};
    bool any() const { return !classes.empty(); }
};

}  // namespace gb
