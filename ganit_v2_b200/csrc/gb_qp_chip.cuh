// PDHG iterations of a diagonal-plus-low-rank QP with few rows, a whole check
// period in one cooperative launch.
//
// The streaming path runs an iteration as five dependent launches (F^T x
// partials, their sum, Q x, primal step, dual step), 19 us on 8,000 assets and
// 29-33 us on 100,000 although every byte is in L2: launch latency.  Here one
// CTA per SM owns kFtxGrid / 148 = 4 consecutive slices of columns (the slices
// of k_ftx_partial) with their rows of F in shared memory, and an iteration is
//   columns   t = F^T x and the rows' sums arrive; Q x, primal step, xbar; then
//             the slices' partials of F^T x+
//   sums      t entry by entry (one CTA each) from the partials, next to the
//             row blocks of A xbar (one slot each; in FP64 the rows' sums are
//             entries of t, with a partial per CTA)
// with no barrier: every exchanged word carries the iteration's tag and its
// reader asks again until it is there.  One buffer of each is enough where a
// writer's next value depends on every reader's last (partials: on all of t; t:
// on all partials, sent after t was read; xbar: on all slots, formed after xbar
// was read); the slots have two, by parity: a block's next slot depends on its
// own columns' CTAs alone, but the one after on a t that all CTAs fed since.
// The dual step of the few rows is taken by every CTA for itself, from the same
// slots in the same order; CTA 0 writes it back.
// Sums are taken in the streaming kernels' order (slices and thread groups of
// k_ftx_partial, lanes of k_ftx_final, columns of F in order, row blocks of A
// as spmv_run takes them), so FP32 iterates keep their bits.  FP64 A^T rows
// are summed in entry order; FP64 rows of F beyond the shared memory (a
// 100,000 x 50 F is 40 MB, the SMs' shared memories hold ~31) come from L2: read
// early, one warp per row, and summed by shuffles.
//
// What bounds it (100,000 x 50, FP64, ~20 K cycles an iteration): the two reads
// of F from shared memory and their FP64 chains (13 K), then three trips of the
// words through L2.  8,009 x 33 is the trips alone: 9 % of the shared-memory
// wavefronts, warps waiting for words.
// Measured on B200, us an iteration of solves of 2,048 iterations, checks
// included, streaming -> here: 100,000 x 50 FP64 32.8 -> 12.4, 8,009 x 33 mixed
// 18.5 -> 6.7.  Of the iterations alone (11.7 and 6.0 us): with two grid barriers
// an iteration in place of the tags 12.7 and 7.0; with the last arrival of a chunk
// running the dual step, and x and bounds read behind the barrier, 16 and 10.
// Reading F once (a warp per four columns, partials by transposing shuffles) took
// 20.4 and 7.0 us against 14.5 and 8.1 at that point: the shuffles cost more than
// the second read saves.
#pragma once
#include "gb_qp.cuh"
#include "gb_resident.cuh"

namespace gb {

constexpr int kQpThreads = 1024;
constexpr int kQpGrid = 148;                     // one CTA per SM
constexpr int kQpPer = kFtxGrid / kQpGrid;       // slices per CTA
static_assert(kQpPer * kQpGrid == kFtxGrid && kQpPer * kThreads == kQpThreads, "a thread group per slice");
constexpr int kQpMaxRows = 4;                    // rows of A
constexpr int kQpOvf = 5;                        // FP64 rows of F per warp read from L2
constexpr int kQpMaxSlots = 256;                 // row blocks of A + kQpMaxRows
constexpr int kQpBarrierTries = 1 << 22;

template <class M, class V>
struct QpArgs {
    int n, m, k, iters;
    int rows_per;            // columns per slice
    int smem_rows;           // of a slice's columns, how many have their row of F in shared memory
    const V* F; const V* D;
    const V* c; const V* l; const V* u; const V* lo; const V* hi;
    const int* at_ptr; const int* at_idx; const M* at_val;
    const unsigned char* at_lg; // log2 lanes per row of A^T (FP32 order); nullptr: entry order
    CsrView<M> A;
    // sums of A's row blocks, then of the rows of STREAM blocks: tagged doubles,
    // one set per parity of the tag
    unsigned long long* slots;
    int slot0[kQpMaxRows], nslots[kQpMaxRows], total_slots;
    unsigned long long used[(kQpMaxSlots + 63) / 64];  // slots that a row's sum reads
    const V* x0; const V* y0;
    V* x; V* y;              // iterate out
    unsigned long long* xbar;   // tagged, by column (FP32)
    V* sumx; V* sumy;
    unsigned long long* part;   // tagged doubles
    unsigned long long* t;
    const SolveState* st;
    SolveState* st_rw;
    unsigned* sync;          // {exits (zero between launches), tag base}
    int* error;
};

// Arrival of this CTA and wait for all CTAs' (the count only grows within a launch).
__device__ __forceinline__ void grid_barrier(unsigned* count, unsigned target, bool& lost) {
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        if (!lost) {
            lost = true;
            for (int k = 0; k < kQpBarrierTries; ++k) {
                unsigned v;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
                if (v >= target) {
                    lost = false;
                    break;
                }
            }
        }
    }
    __syncthreads();
}
// A value and its tag to / from L2.
__device__ __forceinline__ void put_tagged(unsigned long long* p, float v, unsigned tag) {
    const unsigned long long w = static_cast<unsigned long long>(tag) << 32 | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ void put_tagged(unsigned long long* p, double v, unsigned tag) {
    const unsigned long long b = __double_as_longlong(v), t = static_cast<unsigned long long>(tag) << 32;
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(t | (b & 0xffffffffull)), "l"(t | (b >> 32))
                 : "memory");
}
__device__ __forceinline__ bool get_tagged(const unsigned long long* p, unsigned tag, float& v) {
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
    v = __uint_as_float(static_cast<unsigned>(w));
    return static_cast<unsigned>(w >> 32) == tag;
}
__device__ __forceinline__ bool get_tagged(const unsigned long long* p, unsigned tag, double& v) {
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    v = __longlong_as_double((b << 32) | (a & 0xffffffffull));
    return static_cast<unsigned>(a >> 32) == tag && static_cast<unsigned>(b >> 32) == tag;
}
constexpr int kTagTries = 1 << 21;
// Waits for the entry of `tag`; after kTagTries tries sets `lost` (and then waits no more).
template <class V>
__device__ __forceinline__ V wait_tagged(const unsigned long long* p, unsigned tag, bool& lost) {
    V v;
    for (int k = lost ? kTagTries : 0; !get_tagged(p, tag, v); )
        if (++k > kTagTries) {
            lost = true;
            break;
        }
    return v;
}
__device__ __forceinline__ void bar_256(int id) { asm volatile("bar.sync %0, 256;" ::"r"(id) : "memory"); }

// Sum of row block b of A by threads 0..255 into its slot(s) (xbar through
// L2: other CTAs wrote it).  pi / pv: the thread's first entries,
// loaded early.
constexpr int kQpAhead = kChunkNnz / kThreads;
template <class M, class V>
__device__ __forceinline__ void qp_row_block(const QpArgs<M, V>& a, const RowBlock& b, int slot,
                                             const int (&pi)[kQpAhead], const M (&pv)[kQpAhead], V* red, unsigned tag,
                                             bool& lost) {
    constexpr int kW = sizeof(V) / 4;  // words of a tagged xbar entry
    unsigned long long* slots = a.slots + (tag & 1u) * 2 * kQpMaxSlots;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    if (b.kind == kStream) {  // at most kQpMaxRows rows: 32 lanes each (reduce_rows)
        if (wid < b.r1 - b.r0) {
            const int r = b.r0 + wid, p1 = a.A.ptr[r + 1];
            V acc = V(0);
            for (int p = a.A.ptr[r] + lane; p < p1; p += 32)
                acc += static_cast<V>(a.A.val[p]) * wait_tagged<V>(a.xbar + kW * a.A.idx[p], tag, lost);
            acc = warp_sum(acc);
            if (lane == 0) put_tagged(slots + 2 * (a.A.nb + r), double(acc), tag);
        }
        return;
    }
    V acc = V(0), x[kQpAhead];  // long_block
    bool ok[kQpAhead];
#pragma unroll
    for (int i = 0; i < kQpAhead; ++i) ok[i] = b.p0 + tid + i * kThreads >= b.p1 || get_tagged(a.xbar + kW * pi[i], tag, x[i]);
#pragma unroll
    for (int i = 0; i < kQpAhead; ++i)
        if (!ok[i]) x[i] = wait_tagged<V>(a.xbar + kW * pi[i], tag, lost);
#pragma unroll
    for (int i = 0; i < kQpAhead; ++i)
        if (b.p0 + tid + i * kThreads < b.p1) acc += static_cast<V>(pv[i]) * x[i];
    for (int p = b.p0 + tid + kQpAhead * kThreads; p < b.p1; p += kThreads)
        acc += static_cast<V>(a.A.val[p]) * wait_tagged<V>(a.xbar + kW * a.A.idx[p], tag, lost);
    acc = warp_sum(acc);
    if (lane == 0) red[wid] = acc;
    bar_256(1);
    if (tid == 0) {
        V t = V(0);
        for (int w = 0; w < kWarps; ++w) t += red[w];
        put_tagged(slots + 2 * slot, double(t), tag);
    }
    bar_256(1);
}

template <class M, class V>
__global__ void __launch_bounds__(kQpThreads) k_qp_chip(const __grid_constant__ QpArgs<M, V> a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr bool kOvf = sizeof(V) == 8;  // FP64: orders are free, and rows of F may lie outside shared memory
    __shared__ double ts[kMaxRank + kQpMaxRows];
    __shared__ double sh[kQpThreads];
    __shared__ double dots[kQpOvf * kQpThreads / 32];
    __shared__ double sl[kQpMaxSlots];
    __shared__ double fin[kOvf ? 1 : 32 * ((kFtxGrid + 31) / 32)];
    __shared__ double rowp[kOvf ? kQpMaxRows : 1][kQpThreads / 32];
    __shared__ V red[kWarps], ys[kQpMaxRows], sys[kQpMaxRows];
    const SolveState& s = *a.st;
    if (s.active == 0) return;  // every CTA
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int k = a.k, ks = k | 1;                       // odd stride: no bank conflicts between rows
    const int c0 = min(a.n, static_cast<int>(blockIdx.x) * kQpPer * a.rows_per);
    const int nc = min(a.n, c0 + kQpPer * a.rows_per) - c0;  // <= kQpThreads: a column per thread
    const int rp = a.rows_per, rs = a.smem_rows;         // columns per slice, those in shared memory
    const int ro = rp - rs;
    V* fs = reinterpret_cast<V*>(smem);                  // kQpPer x rs rows of F
    V* xs = fs + static_cast<size_t>(kQpPer) * rs * ks;  // the CTA's columns of x
    for (int e = tid; e < nc * k; e += kQpThreads) {
        const int r = e / k, c = e - r * k, q = r / rp, i = r - q * rp;
        if (i < rs) fs[static_cast<size_t>(q * rs + i) * ks + c] = a.F[static_cast<size_t>(c0) * k + e];
    }
    const int j = c0 + tid;                              // this thread's column (tid < nc)
    if (tid < nc) {
        const V v = a.x0[j];
        xs[tid] = v;
        a.x[j] = v;
    }
    if (tid < a.m) {
        ys[tid] = a.y0[tid];
        sys[tid] = a.sumy[tid];
    }
    const V tau = static_cast<V>(s.tau), sigma = static_cast<V>(s.sigma);
    bool lost = false;
    const unsigned base = a.sync[1];
    const int q = tid / kThreads, qt = tid % kThreads;  // slice of the CTA, thread in it (k_ftx_partial)
    const int G = kThreads / k, g = qt / k, c = qt - g * k;
    const int slice = blockIdx.x * kQpPer + q;
    const int my_q = tid / rp, my_i = tid - my_q * rp;  // this thread's column: its slice and place there
    __syncthreads();
    auto partials = [&](unsigned tag) {
        double acc = 0.0;
        const int r1 = min(rp, nc - q * rp);  // rows of this slice
        if (g < G) {
            const V* x = xs + q * rp;
            if constexpr (kOvf) {  // rows outside shared memory first: their L2 latency is paid once
                const V* f = a.F + static_cast<size_t>(c0 + q * rp + rs + g) * k + c;
#pragma unroll 8
                for (int r = rs + g; r < r1; r += G, f += G * k) acc += double(*f) * double(x[r]);
            }
            const V* f = fs + (q * rs + g) * ks + c;
            const int e = min(r1, rs), step = G * ks;
#pragma unroll 8
            for (int r = g; r < e; r += G, f += step) acc += double(*f) * double(x[r]);
        }
        sh[tid] = acc;
        if constexpr (kOvf) {  // one partial per CTA, and the rows' own
            __syncthreads();
            if (tid < 8 * k) {  // entry tid / 8: eight threads fold the groups of every slice
                double t = 0.0;
                for (int z = tid & 7; z < kQpPer * G; z += 8) t += sh[(z / G) * kThreads + (z % G) * k + (tid >> 3)];
                for (int o = 4; o > 0; o >>= 1) t += __shfl_down_sync(0xffu << (lane & 24), t, o, 8);
                if ((tid & 7) == 0) put_tagged(a.part + 2 * ((tid >> 3) * kQpGrid + blockIdx.x), t, tag);
            }
            return;
        }
        bar_256(2 + q);
        if (qt < k) {
            double t = 0.0;
            for (int gg = 0; gg < G; ++gg) t += sh[q * kThreads + gg * k + qt];
            put_tagged(a.part + 2 * (qt * kFtxGrid + slice), t, tag);
        }
    };
    // k_ftx_final of entries [e0, e1), entry e in CTA e: its partials by warps 8
    // and up (FP32: five of the 19 rounds of 32 each), the sum by warp 8.  FP64
    // has a partial per CTA instead of one per slice, and the rows' sums as
    // entries k, k + 1, ...
    constexpr int kParts = kOvf ? kQpGrid : kFtxGrid, kTerm = (kParts + 31) / 32, kAtOnce = 5;
    constexpr int kFinWarps = (kTerm + kAtOnce - 1) / kAtOnce;
    auto finish_t = [&](int e0, int e1, unsigned tag) {
        const int fw = wid - kWarps;
        if (fw < 0 || fw >= kFinWarps) return;
        for (int e = e0 + blockIdx.x; e < e1; e += kQpGrid) {
            const unsigned long long* p = a.part + 2 * static_cast<size_t>(e) * kParts;
            double v[kAtOnce];
            bool ok[kAtOnce];
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i) {
                const int z = lane + 32 * (kAtOnce * fw + i);
                v[i] = 0.0;
                ok[i] = z >= kParts || get_tagged(p + 2 * z, tag, v[i]);
            }
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i) {
                const int z = lane + 32 * (kAtOnce * fw + i);
                if (!ok[i]) v[i] = wait_tagged<double>(p + 2 * z, tag, lost);
            }
            double t = 0.0;
            if constexpr (kFinWarps == 1) {
#pragma unroll
                for (int i = 0; i < kAtOnce; ++i)
                    if (lane + 32 * i < kParts) t += v[i];
            } else {
#pragma unroll
                for (int i = 0; i < kAtOnce; ++i)
                    if (kAtOnce * fw + i < kTerm) fin[32 * (kAtOnce * fw + i) + lane] = v[i];
                asm volatile("bar.sync 6, %0;" ::"n"(32 * kFinWarps) : "memory");
                if (fw == 0) {
#pragma unroll
                    for (int i = 0; i < kTerm; ++i)
                        if (lane + 32 * i < kParts) t += fin[32 * i + lane];
                }
                asm volatile("bar.sync 6, %0;" ::"n"(32 * kFinWarps) : "memory");
            }
            if (fw == 0) {
                t = warp_sum(t);
                if (lane == 0) put_tagged(a.t + 2 * e, t, tag);
            }
        }
    };
    // dual step of row i from its slots (shared memory), the same in every CTA
    auto dual = [&](int i) {
        const int b0 = kOvf ? i : a.slot0[i], nb = kOvf ? 1 : a.nslots[i];
        V t = static_cast<V>(sl[b0]);
        if (nb > 1) {
            t = V(0);
#pragma unroll 8
            for (int z = 0; z < nb; ++z) t += static_cast<V>(sl[b0 + z]);
        }
        const V yi = ys[i];
        const V qv = yi - sigma * t;  // DualEpi
        const V lk = sigma * a.lo[i], hk = sigma * a.hi[i];
        V w = -qv;
        w = (w < lk) ? lk : w;
        w = (hk < w) ? hk : w;
        const V v = qv + w;
        ys[i] = v;
        sys[i] = sys[i] + v;
    };
    partials(base + 1);
    finish_t(0, k, base + 1);
    for (int it = 0;; ++it) {
        const unsigned tag = base + 1 + it;  // of t; the rows' sums of the iteration before have tag - 1 (FP32)
        // the column phase's constants
        V cj = V(0), lj = V(0), uj = V(0), sj = V(0);
        double dj = 0.0;
        int p0 = 0, len = 0;
        if (it < a.iters && tid < nc) {
            cj = a.c[j];
            lj = a.l[j];
            uj = a.u[j];
            sj = a.sumx[j];
            dj = double(a.D[j]);
            p0 = a.at_ptr[j];
            len = a.at_ptr[j + 1] - p0;
        }
        // rows of F outside shared memory: row o = warp + 32 i of the kQpPer x ro,
        // a lane's columns lane and lane + 32
        double f0[kQpOvf], f1[kQpOvf];
        if constexpr (kOvf) {
#pragma unroll
            for (int i = 0; i < kQpOvf; ++i) {
                const int o = wid + 32 * i, oq = ro ? o / ro : kQpPer, r = oq * rp + rs + (o - oq * ro);
                const bool in = it < a.iters && oq < kQpPer && r < min(nc, (oq + 1) * rp);
                const V* f = a.F + static_cast<size_t>(c0 + r) * k + lane;
                f0[i] = in && lane < k ? double(f[0]) : 0.0;
                f1[i] = in && lane + 32 < k ? double(f[32]) : 0.0;
            }
        }
        if (tid < k && it < a.iters) ts[tid] = wait_tagged<double>(a.t + 2 * tid, tag, lost);
        if (kOvf) {
            if (it > 0 && tid >= k && tid < k + a.m) sl[tid - k] = wait_tagged<double>(a.t + 2 * tid, tag, lost);
        } else if (it > 0) {
            // (from the other end: t's threads wait for t)
            for (int z = kQpThreads - 1 - tid; z < a.total_slots; z += kQpThreads)
                if (a.used[z >> 6] >> (z & 63) & 1) sl[z] = wait_tagged<double>(a.slots + ((tag - 1) & 1u) * 2 * kQpMaxSlots + 2 * z, tag - 1, lost);
        }
        __syncthreads();
        if (it > 0 && tid >= kQpThreads - kQpMaxRows && kQpThreads - 1 - tid < a.m) dual(kQpThreads - 1 - tid);
        if (it == a.iters) break;
        if constexpr (kOvf) {
            if (ro) {
                const double t0 = lane < k ? ts[lane] : 0.0, t1 = lane + 32 < k ? ts[lane + 32] : 0.0;
#pragma unroll
                for (int i = 0; i < kQpOvf; ++i) {
                    const double d = warp_sum(f0[i] * t0 + f1[i] * t1);
                    if (lane == 0) dots[wid + 32 * i] = d;
                }
            }
        }
        // the column's entries of A arrive during its dot product
        M av[kQpMaxRows];
        int ai[kQpMaxRows], lgj = 0;
#pragma unroll
        for (int e = 0; e < kQpMaxRows; ++e) {
            av[e] = e < len ? a.at_val[p0 + e] : static_cast<M>(0.0f);
            ai[e] = e < len ? a.at_idx[p0 + e] : 0;
        }
        if (len > 1 && a.at_lg != nullptr) lgj = a.at_lg[j];  // one entry: the same sum either way
        double s0 = 0.0;
        if (tid < nc && my_i < rs) {
            const V* f = fs + (my_q * rs + my_i) * ks;
#pragma unroll 8
            for (int e = 0; e < k; ++e) s0 += double(f[e]) * ts[e];
        }
        __syncthreads();
        V xb = V(0);
        if (tid < nc) {
            if (kOvf && my_i >= rs) s0 = dots[my_q * ro + my_i - rs];
            V pr[kQpMaxRows];
#pragma unroll
            for (int e = 0; e < kQpMaxRows; ++e) pr[e] = e < len ? static_cast<V>(av[e]) * ys[ai[e]] : V(0);
            // one lane per row: entry order; more: the lanes' parts, then the tree
            const V aty = lgj ? ((V(0) + pr[0]) + pr[2]) + ((V(0) + pr[1]) + pr[3])
                              : (((V(0) + pr[0]) + pr[1]) + pr[2]) + pr[3];
            const V xj = xs[tid];
            const V qx = static_cast<V>(2.0 * (s0 + dj * double(xj)));
            const V grad = cj - aty + qx;  // PrimalEpi
            V v = xj - tau * grad;
            v = (v < lj) ? lj : v;
            v = (uj < v) ? uj : v;
            xs[tid] = v;
            a.x[j] = v;
            xb = V(2) * v - xj;
            if (!kOvf) put_tagged(a.xbar + j, xb, tag);
            a.sumx[j] = sj + v;
        }
        if constexpr (kOvf) {  // A xbar over the CTA's columns, row by row
#pragma unroll
            for (int i = 0; i < kQpMaxRows; ++i) {
                if (i >= a.m) break;
                double v = 0.0;
#pragma unroll
                for (int e = 0; e < kQpMaxRows; ++e)
                    if (e < len && ai[e] == i) v += static_cast<double>(av[e]) * static_cast<double>(xb);
                v = warp_sum(v);
                if (lane == 0) rowp[i][wid] = v;
            }
        }
        __syncthreads();
        if (kOvf && wid < a.m) {
            const double v = warp_sum(rowp[wid][lane]);
            if (lane == 0) put_tagged(a.part + 2 * ((k + wid) * kQpGrid + blockIdx.x), v, tag + 1);
        }
        if (it + 1 < a.iters) partials(tag + 1);
        if constexpr (kOvf) {  // FP64: t is all the sums there are
            finish_t(it + 1 < a.iters ? 0 : k, k + a.m, tag + 1);
            continue;
        }
        // the row phase's first entries
        int pi[kQpAhead];
        M pv[kQpAhead];
        const bool rows = tid < kThreads && static_cast<int>(blockIdx.x) < a.A.nb;
        auto ahead = [&](int at) {
            const int p0 = a.A.blocks[at].p0 + tid, p1 = a.A.blocks[at].p1;
#pragma unroll
            for (int i = 0; i < kQpAhead; ++i) {
                pi[i] = p0 + i * kThreads < p1 ? a.A.idx[p0 + i * kThreads] : 0;
                pv[i] = p0 + i * kThreads < p1 ? a.A.val[p0 + i * kThreads] : static_cast<M>(0.0f);
            }
        };
        if (rows) {
            ahead(blockIdx.x);
            for (int at = blockIdx.x;;) {
                qp_row_block(a, a.A.blocks[at], at, pi, pv, red, tag, lost);
                at += kQpGrid;
                if (at >= a.A.nb) break;
                ahead(at);
            }
        } else if (tid >= kThreads && it + 1 < a.iters) {
            finish_t(0, k, tag + 1);
        }
    }
    lost = __syncthreads_or(lost);
    if (blockIdx.x == 0 && tid < a.m) {
        a.y[tid] = ys[tid];
        a.sumy[tid] = sys[tid];
    }
    if (tid == 0) {
        if (lost) {  // the solve stops at the coming check and reports the error
            atomicExch(a.error, 1);
            a.st_rw->max_iter = 0;
        }
        __threadfence();
        if (atomicAdd(a.sync, 1u) == kQpGrid - 1) {  // every CTA has read the base
            a.sync[0] = 0u;
            a.sync[1] = base + static_cast<unsigned>(a.iters) + 1u;
        }
    }
}

// Columns of a slice whose row of F fits in shared memory (next to x); the
// others must fit the registers.  0: does not fit.
// dynamic shared memory; the kernel's static arrays take ~14 KB, in FP32 ~19
template <class V>
constexpr size_t kQpSmem = (sizeof(V) == 8 ? 213 : 207) * size_t(1024);
template <class V>
inline int qp_smem_rows(int n, int k, int* rows_per) {
    *rows_per = div_up(n, kFtxGrid);
    const int nc = kQpPer * *rows_per;
    if (nc > kQpThreads) return 0;
    const size_t row = sizeof(V) * (k | 1), x = sizeof(V) * nc;
    const int rs = static_cast<int>(std::min<size_t>(*rows_per, (kQpSmem<V> - x) / (kQpPer * row)));
    if (rs == *rows_per) return rs;
    return sizeof(V) == 8 && k <= 64 && kQpPer * (*rows_per - rs) <= kQpOvf * kQpThreads / 32 ? rs : 0;
}

}  // namespace gb
