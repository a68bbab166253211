// On-chip PDHG iterations of one LP that a cluster cannot hold: the whole GPU
// keeps it, one CTA per SM, a check period per cooperative launch.
//
// The streaming kernels take two dependent launches and a pass over the matrix
// in L2 per iteration: 13.7 us on a blending LP of 411K nonzeros in FP64,
// 17.0 us at 2.9M in FP32.  Here every CTA owns a contiguous share of A^T's
// rows and of A's rows (by nonzeros) with its matrix entries, vectors and
// iterate in shared memory.  The entries of y and xbar that its rows gather --
// for an LP with any locality a small part -- are listed once; every half
// iteration the CTA copies them from L2 into shared memory and gathers there
// through 16-bit local positions.  Packing, lanes per row and so the FP32 bits
// are k_resident's; slices that do not fit the shared memory are read from L2.
//
// No barrier separates the halves: an entry travels with the iteration's tag
// (FP32: value and tag in one 64-bit word, FP64: two words, each half with the
// tag; a 64-bit access is never torn), and a reader asks again until the tag is
// there.  A CTA thus waits for the entries it needs and no others.  Entries
// live in rings of kGridRing slots; a grid barrier every kGridRing - 1
// iterations keeps a writer from reaching a slot that is still read (between
// two barriers at most kGridRing consecutive y's are alive).
//
// What bounds it: two trips through L2 per iteration at small sizes; at 2.9M
// nonzeros the shared-memory wavefronts of the sums and the 40 % of the matrix
// that comes from L2.  Measured on B200, us an iteration of solves of 2,048
// iterations, checks included, streaming -> here: blending 120K nonzeros FP64
// 8.7 -> 4.0, 411K FP64 13.7 -> 4.8, 2.9M FP32 17.0 -> 10.0; random 6000 x 15001
// (no locality) FP64 9.5 -> 5.7, FP32 7.7 -> 5.9.  With two grid barriers an
// iteration in place of the tags the three blending LPs took 1.44, 1.25 and 1.11
// times as long, the random one 0.97 times.
#pragma once
#include "gb_qp_chip.cuh"
#include "gb_resident.cuh"

namespace gb {

constexpr int kGridThreads = 1024;
constexpr int kGridCtas = 148;
constexpr size_t kGridSmem = 226 * 1024;
constexpr int kGridRing = 8;
constexpr int kGridTries = 1 << 21;

struct GridCta {
    int slice0, ns_t, ns_a;
    int res_t, res_a;          // slices of either side whose pairs are in shared memory (the first ones)
    int pairs_t, pairs_a;      // pairs of those
    int own_t, own_a;
    int pos_t0, pos_a0;        // first packed position of its columns / rows
    int u_t, u_a;              // entries of y / xbar it gathers
    int list_t0, list_a0;      // where their packed positions are listed
    long long pair_t0, pair_a0;  // first pair of either side in the packed arrays
};

template <class V>
inline size_t grid_fixed_bytes(const GridCta& c) {
    auto r4 = [](int k) { return static_cast<size_t>((k + 3) & ~3); };
    return sizeof(V) * (r4(c.u_a + 1) + r4(c.u_t + 1) + 5 * r4(c.own_t) + 4 * r4(c.own_a)) +
           16 * static_cast<size_t>(c.ns_t + c.ns_a);
}

template <class M, class V>
struct GridArgs {
    const GridCta* cta;
    const ResSlice* slices;
    const unsigned* idx;
    const M* val;
    const int* list_t; const int* list_a;  // packed positions of the gathered rows / columns
    const int* col_at; const int* row_at;  // packed position -> column / row
    unsigned long long* xg;                // rings of xbar and y by packed position, with tags
    unsigned long long* yg;
    int n, m;
    const V* x0; const V* y0;
    V* x; V* y; V* sumx; V* sumy;
    const V* c; const V* l; const V* u; const V* lo; const V* hi;
    SolveState* st;
    unsigned* sync;
    int* error;
    int iters;
};

template <class M, class V>
__global__ void __launch_bounds__(kGridThreads) k_grid(const __grid_constant__ GridArgs<M, V> a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const SolveState& s = *a.st;
    if (s.active == 0) return;  // every CTA
    const GridCta r = a.cta[blockIdx.x];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int T = kGridThreads, W = T / 32;
    constexpr size_t kW = sizeof(V) / 4;  // words of a tagged entry
    const unsigned base = a.sync[2];      // tags of this launch: base + 1 + iteration
    auto r4 = [](int k) { return (k + 3) & ~3; };
    V* xs = reinterpret_cast<V*>(smem);
    V* ys = xs + r4(r.u_a + 1);
    V* ox = ys + r4(r.u_t + 1);
    V* oc = ox + r4(r.own_t);
    V* ol = oc + r4(r.own_t);
    V* ou = ol + r4(r.own_t);
    V* osx = ou + r4(r.own_t);
    V* oy = osx + r4(r.own_t);
    V* olo = oy + r4(r.own_a);
    V* ohi = olo + r4(r.own_a);
    V* osy = ohi + r4(r.own_a);
    ResSlice* sl = reinterpret_cast<ResSlice*>(osy + r4(r.own_a));
    unsigned* idx = reinterpret_cast<unsigned*>(sl + r.ns_t + r.ns_a);
    M* val = reinterpret_cast<M*>(idx + 32 * (r.pairs_t + r.pairs_a));
    for (int k = tid; k < r.ns_t + r.ns_a; k += T) cp_async16(sl + k, a.slices + r.slice0 + k);
    constexpr int kPer16 = 16 / static_cast<int>(sizeof(M));
    auto fetch = [&](int at, int pairs, long long from) {
        for (int k = tid; k < 8 * pairs; k += T) cp_async16(idx + 32 * at + 4 * k, a.idx + 32 * from + 4 * k);
        for (int k = tid; k < 64 / kPer16 * pairs; k += T)
            cp_async16(val + 64 * at + kPer16 * k, a.val + 64 * from + kPer16 * k);
    };
    fetch(0, r.pairs_t, r.pair_t0);
    fetch(r.pairs_t, r.pairs_a, r.pair_a0);
    for (int k = tid; k < r.own_t; k += T) {
        const int j = a.col_at[r.pos_t0 + k];
        ox[k] = a.x0[j];
        oc[k] = a.c[j];
        ol[k] = a.l[j];
        ou[k] = a.u[j];
        osx[k] = a.sumx[j];
    }
    for (int k = tid; k < r.own_a; k += T) {
        const int i = a.row_at[r.pos_a0 + k];
        const V v = a.y0[i];
        oy[k] = v;
        put_tagged(a.yg + kW * (r.pos_a0 + k), v, base + 1);
        olo[k] = a.lo[i];
        ohi[k] = a.hi[i];
        osy[k] = a.sumy[i];
    }
    if (tid == 0) {
        xs[r.u_a] = V(0);
        ys[r.u_t] = V(0);
    }
    const V tau = static_cast<V>(s.tau), sigma = static_cast<V>(s.sigma);
    cp_async_wait_all();
    bool lost = false;
    unsigned target = 0;
    // The gathered entries of a ring slot into `to`, each once its tag is there.
    constexpr int kAhead = sizeof(V) == 4 ? 4 : 2;  // entries a thread asks for at once
    auto collect = [&](V* to, const unsigned long long* from, const int* list, int u, unsigned tag) {
        for (int k0 = tid; k0 < u; k0 += kAhead * T) {
            int at[kAhead];  // -1: taken
#pragma unroll
            for (int i = 0; i < kAhead; ++i) at[i] = k0 + i * T < u ? list[k0 + i * T] : -1;
            int tries = lost ? kGridTries : 0;
            for (bool open = true; open;) {
                V v[kAhead];
                bool ok[kAhead];
#pragma unroll
                for (int i = 0; i < kAhead; ++i) ok[i] = at[i] >= 0 && get_tagged(from + kW * at[i], tag, v[i]);
                open = false;
#pragma unroll
                for (int i = 0; i < kAhead; ++i) {
                    if (ok[i]) {
                        to[k0 + i * T] = v[i];
                        at[i] = -1;
                    }
                    open |= at[i] >= 0;
                }
                if (open && ++tries > kGridTries) {
                    lost = true;
                    break;
                }
            }
        }
        __syncthreads();
    };
    __syncthreads();
    for (int it = 0; it < a.iters; ++it) {
        const int slot = it % kGridRing;
        const unsigned tag = base + 1 + it;
        if (it > 0 && it % (kGridRing - 1) == 0) grid_barrier(a.sync, target += kGridCtas, lost);
        collect(ys, a.yg + kW * slot * a.m, a.list_t + r.list_t0, r.u_t, tag);
        for (int q = warp; q < r.ns_t; q += W) {  // primal half (PrimalEpi)
            const ResSlice e = sl[q];
            const int np = e.meta & 0xff, lg = (e.meta >> 8) & 0xf, nr = e.meta >> 12, grp = min(lane >> lg, nr - 1);
            const int k = e.own0 + grp;
            const V xk = ox[k], ck = oc[k], lk = ol[k], uk = ou[k], sk = osx[k];
            const V t = q < r.res_t
                            ? slice_sum<M, V>(e.pair0, np, lg, idx, val, ys, lane)
                            : slice_sum<M, V>(e.pair0, np, lg, a.idx + 32 * r.pair_t0, a.val + 64 * r.pair_t0, ys, lane);
            const V g = ck - t + V(0);
            V v = xk - tau * g;
            v = (v < lk) ? lk : v;
            v = (uk < v) ? uk : v;
            if ((lane & ((1 << lg) - 1)) == 0 && (lane >> lg) < nr) {
                ox[k] = v;
                osx[k] = sk + v;
                put_tagged(a.xg + kW * (static_cast<size_t>(slot) * a.n + r.pos_t0 + k), V(2) * v - xk, tag);
            }
        }
        collect(xs, a.xg + kW * slot * a.n, a.list_a + r.list_a0, r.u_a, tag);
        const size_t next = static_cast<size_t>((it + 1) % kGridRing) * a.m;
        for (int q = warp; q < r.ns_a; q += W) {  // dual half (DualEpi)
            const ResSlice e = sl[r.ns_t + q];
            const int np = e.meta & 0xff, lg = (e.meta >> 8) & 0xf, nr = e.meta >> 12, grp = min(lane >> lg, nr - 1);
            const int k = e.own0 + grp;
            const V yk = oy[k], sk = osy[k], lk = sigma * olo[k], hk = sigma * ohi[k];
            const V t = q < r.res_a
                            ? slice_sum<M, V>(e.pair0, np, lg, idx + 32 * r.pairs_t, val + 64 * r.pairs_t, xs, lane)
                            : slice_sum<M, V>(e.pair0, np, lg, a.idx + 32 * r.pair_a0, a.val + 64 * r.pair_a0, xs, lane);
            const V qv = yk - sigma * t;
            V w = -qv;
            w = (w < lk) ? lk : w;
            w = (hk < w) ? hk : w;
            const V v = qv + w;
            if ((lane & ((1 << lg) - 1)) == 0 && (lane >> lg) < nr) {
                osy[k] = sk + v;
                oy[k] = v;
                put_tagged(a.yg + kW * (next + r.pos_a0 + k), v, tag + 1);
            }
        }
    }
    __syncthreads();
    for (int k = tid; k < r.own_t; k += T) {
        const int j = a.col_at[r.pos_t0 + k];
        a.x[j] = ox[k];
        a.sumx[j] = osx[k];
    }
    for (int k = tid; k < r.own_a; k += T) {
        const int i = a.row_at[r.pos_a0 + k];
        a.y[i] = oy[k];
        a.sumy[i] = osy[k];
    }
    lost = __syncthreads_or(lost);
    if (tid == 0) {
        if (lost) {  // the solve stops at the coming check and reports the error
            atomicExch(a.error, 1);
            a.st->max_iter = 0;
        }
        __threadfence();
        if (atomicAdd(a.sync + 1, 1u) == kGridCtas - 1) {  // every CTA has passed its last barrier
            a.sync[0] = 0u;
            a.sync[1] = 0u;
            a.sync[2] = base + static_cast<unsigned>(a.iters) + 1u;
        }
    }
}

// ---------------------------------------------------------------- packing
// Distinct entries of the gathered vector that rows [row0, row1) of each CTA
// reference: a bitmap of the vector per CTA (global scratch, `words` words),
// its running counts, and the number of entries.
static __global__ void __launch_bounds__(1024) k_grid_mark(const ResSide* __restrict__ sides, const int* __restrict__ ptr,
                                                           const int* __restrict__ idx, int words,
                                                           unsigned* __restrict__ bits, int* __restrict__ before,
                                                           int* __restrict__ count) {
    __shared__ int part[32];
    const ResSide& sd = sides[blockIdx.x];
    unsigned* b = bits + static_cast<size_t>(blockIdx.x) * words;
    int* f = before + static_cast<size_t>(blockIdx.x) * words;
    for (int p = ptr[sd.row0] + threadIdx.x; p < ptr[sd.row1]; p += 1024) atomicOr(b + (idx[p] >> 5), 1u << (idx[p] & 31));
    __threadfence();
    __syncthreads();
    const int per = (words + 1023) / 1024, w0 = min(words, static_cast<int>(threadIdx.x) * per), w1 = min(words, w0 + per);
    int n = 0;
    for (int w = w0; w < w1; ++w) n += __popc(__ldcg(b + w));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int inc = n;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    if (lane == 31) part[wid] = inc;
    __syncthreads();
    if (wid == 0) {
        int v = part[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int z = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += z;
        }
        part[lane] = v;
    }
    __syncthreads();
    int run = inc - n + (wid ? part[wid - 1] : 0);
    for (int w = w0; w < w1; ++w) {
        f[w] = run;
        run += __popc(__ldcg(b + w));
    }
    if (threadIdx.x == 1023) count[blockIdx.x] = run;
}
// The lists: packed position (`pos` of the gathered vector) of every marked entry.
static __global__ void k_grid_lists(int words, const unsigned* __restrict__ bits, const int* __restrict__ before,
                                    const int* __restrict__ list0, const int* __restrict__ pos, int* __restrict__ list) {
    const unsigned* b = bits + static_cast<size_t>(blockIdx.x) * words;
    const int* f = before + static_cast<size_t>(blockIdx.x) * words;
    for (int w = threadIdx.x; w < words; w += blockDim.x) {
        int k = list0[blockIdx.x] + f[w];
        for (unsigned m = b[w]; m; m &= m - 1) list[k++] = pos[32 * w + __ffs(m) - 1];
    }
}
// Local positions of every entry, at its slot (k_res_entries' arithmetic).
static __global__ void k_grid_entries(const ResSide* __restrict__ sides, const int* __restrict__ ptr,
                                      const int* __restrict__ col, const int* __restrict__ slot,
                                      const ResSliceAt* __restrict__ slices, int words,
                                      const unsigned* __restrict__ bits, const int* __restrict__ before,
                                      unsigned short* __restrict__ idx) {
    const ResSide& sd = sides[blockIdx.x];
    const unsigned* b = bits + static_cast<size_t>(blockIdx.x) * words;
    const int* f = before + static_cast<size_t>(blockIdx.x) * words;
    for (int r = sd.row0 + threadIdx.x; r < sd.row1; r += blockDim.x) {
        const int sr = slot[r];
        const ResSliceAt e = slices[sr >> 5];
        const int lg = (e.meta >> 8) & 0xf, G = 1 << lg, p0 = ptr[r], len = ptr[r + 1] - p0;
        for (int k = 0; k < len; ++k) {
            const int t = k >> lg, lane = ((sr & 31) << lg) + (k & (G - 1)), c = col[p0 + k], w = c >> 5;
            idx[(e.pair0 + (t >> 1)) * 64 + 2 * lane + (t & 1)] =
                static_cast<unsigned short>(f[w] + __popc(b[w] & ((1u << (c & 31)) - 1u)));
        }
    }
}
static __global__ void k_grid_inverse(int k, const int* __restrict__ at, int* __restrict__ pos) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < k; q += gridDim.x * blockDim.x) pos[at[q]] = q;
}
// Padding of a CTA's pairs: the zero slot after its gathered entries.
static __global__ void k_grid_fill(const long long* __restrict__ pair0, const int* __restrict__ count, unsigned* __restrict__ idx) {
    const unsigned z = static_cast<unsigned>(count[blockIdx.x]) * 0x10001u;
    for (long long k = 32 * pair0[blockIdx.x] + threadIdx.x; k < 32 * pair0[blockIdx.x + 1]; k += blockDim.x) idx[k] = z;
}

struct GridPlan {
    bool built = false, on = false;
    DevBuf<unsigned char> mem[2];                  // everything below but the values
    GridCta* cta = nullptr;
    ResSlice* slices = nullptr;
    ResSliceAt* at = nullptr;
    ResSide* sides[2] = {};                        // A^T, A
    int *list[2] = {}, *src[2] = {}, *slot[2] = {}, *pos[2] = {};
    unsigned* bits[2] = {};                        // packing alone: in Problem::plan_scratch, as `before`
    int *before[2] = {}, *count[2] = {}, *list0[2] = {};
    unsigned char* lg[2] = {};
    long long* pair0[2] = {};
    unsigned* idx = nullptr;
    unsigned long long *gx = nullptr, *gy = nullptr;  // rings of xbar / y by packed position
    unsigned* sync = nullptr;
    DevBuf<float> val32;
    DevBuf<double> val64;
    DevBuf<__nv_bfloat16> valbf;
    size_t smem = 0;
    long long pairs = 0;
};

}  // namespace gb
