// Host-only checker of the on-chip plan (ganit_v2_b200/csrc/gb_resident.cuh),
// compiled and run by tests/test_resident.py; no GPU involved.  For random
// matrices it deals an instance's slices to clusters of 1..16 CTAs, follows
// the packing kernels' index arithmetic on the host, and checks that every
// position and every packed entry is written once and inside its CTA's share
// and that a slice's sums are bit for bit the streaming kernels' FP32 sums.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "../ganit_v2_b200/csrc/gb_resident.cuh"

using namespace gb;

static int fail(const char* what, const std::string& name, int C) {
    std::printf("FAIL %s C=%d: %s\n", name.c_str(), C, what);
    return 1;
}

struct Mat {
    int rows, cols;
    std::vector<int> ptr, idx;
    std::vector<float> val;
};

static Mat random_mat(int rows, int cols, int kmin, int kmax, std::mt19937& rng) {
    Mat A{rows, cols, {0}, {}, {}};
    std::normal_distribution<float> N;
    for (int i = 0; i < rows; ++i) {
        const int k = std::min<int>(cols, kmin + rng() % (kmax - kmin + 1));
        for (int e = 0; e < k; ++e) {
            A.idx.push_back(rng() % cols);
            A.val.push_back(N(rng));
        }
        A.ptr.push_back(static_cast<int>(A.idx.size()));
    }
    return A;
}

// lanes' parts, then the shuffle tree, of one row (reduce_rows)
static float group_sum(const std::vector<float>& prod, int lg) {
    const int G = 1 << lg;
    std::vector<float> acc(G, 0.0f);
    for (int g = 0; g < G; ++g)
        for (size_t k = g; k < prod.size(); k += G) acc[g] += prod[k];
    for (int o = G >> 1; o > 0; o >>= 1)
        for (int g = 0; g + o < G; ++g) acc[g] += acc[g + o];  // lane g reads the old value of lane g + o
    return acc[0];
}

static int check(const std::string& name, const Mat& T, const Mat& A, bool by_block, int C) {
    const Mat* mats[2] = {&T, &A};
    std::array<ResHist, 2> H;
    std::vector<unsigned char> lg_of[2];
    for (int sd = 0; sd < 2; ++sd) {
        const Mat& M = *mats[sd];
        lg_of[sd].resize(M.rows);
        const Schedule s = build_schedule(M.ptr.data(), M.rows);
        for (const RowBlock& b : s.blocks) {
            if (b.kind != kStream) return fail("test matrix has long rows", name, C);
            if (!res_hist_rows(M.ptr.data(), b.r0, b.r1, by_block ? b.lg : -1, H[sd])) return fail("histogram", name, C);
            for (int r = b.r0; r < b.r1; ++r)
                lg_of[sd][r] = by_block ? b.lg : res_lg64(M.ptr[r + 1] - M.ptr[r]);
        }
        H[sd].count();
    }
    ResDeal D;
    res_deal(H, C, D);
    ResTables tab;
    tab.pairs = 3;  // tables do not start at 0
    tab.add(0, H, D, 0, T.rows, 0, A.rows);
    std::vector<int> pos[2], slot[2];
    for (int sd = 0; sd < 2; ++sd) {  // k_res_rank
        const Mat& M = *mats[sd];
        const ResSide& S = tab.sides[sd][0];
        int next[6][kResBins];
        std::memcpy(next, S.rank0, sizeof next);
        pos[sd].assign(M.rows, -1);
        slot[sd].assign(M.rows, -1);
        const int npos = sd == 0 ? D.cta[0].n : D.cta[0].m;
        std::vector<char> seen(npos, 0);
        for (int r = 0; r < M.rows; ++r) {
            const int len = M.ptr[r + 1] - M.ptr[r], lg = lg_of[sd][r], steps = (len + (1 << lg) - 1) >> lg;
            const int k = next[lg][(steps + 1) >> 1]++, rows = 32 >> lg;
            const int e = S.slice0[lg] + k / rows, grp = k % rows;
            if (S.slice0[lg] < 0 || e >= static_cast<int>(tab.at.size())) return fail("slice entry", name, C);
            const ResSliceAt& at = tab.at[e];
            if (((at.meta >> 8) & 0xf) != lg || grp >= (at.meta >> 12)) return fail("slice of the wrong kind", name, C);
            if (2 * (at.meta & 0xff) < steps) return fail("row longer than its slice", name, C);
            pos[sd][r] = at.pos0 + grp;
            slot[sd][r] = e * 32 + grp;
            if (pos[sd][r] < 0 || pos[sd][r] >= npos || seen[pos[sd][r]]++) return fail("positions", name, C);
        }
    }
    long long used = 0;
    std::vector<float> val(static_cast<size_t>(tab.pairs) * 64, 0.0f);
    std::vector<int> idx(val.size(), -1);
    for (int sd = 0; sd < 2; ++sd)  // k_res_entries / k_res_values
        for (int r = 0; r < mats[sd]->rows; ++r) {
            const ResSliceAt& at = tab.at[slot[sd][r] >> 5];
            const int lg = (at.meta >> 8) & 0xf, p0 = mats[sd]->ptr[r], len = mats[sd]->ptr[r + 1] - p0;
            for (int k = 0; k < len; ++k) {
                const int t = k >> lg, lane = ((slot[sd][r] & 31) << lg) + (k & ((1 << lg) - 1));
                const long long w = (at.pair0 + (t >> 1)) * 64 + 2 * lane + (t & 1);
                if (lane >= 32 || w < 3 * 64 || w >= static_cast<long long>(idx.size()) || idx[w] >= 0)
                    return fail("packed entry", name, C);
                idx[w] = pos[1 - sd][mats[sd]->idx[p0 + k]];
                val[w] = mats[sd]->val[p0 + k];
                ++used;
            }
        }
    if (used != T.ptr.back() + A.ptr.back()) return fail("entry count", name, C);
    // every CTA's slices, as k_resident runs them
    std::mt19937 rng(5);
    std::normal_distribution<float> N;
    std::vector<float> g[2] = {std::vector<float>(A.rows), std::vector<float>(T.rows)};  // y, xbar (source order)
    for (auto& v : g)
        for (float& x : v) x = N(rng);
    int slices = 0;
    std::vector<int> got[2] = {std::vector<int>(T.rows, 0), std::vector<int>(A.rows, 0)};
    std::vector<int> row_at[2] = {std::vector<int>(D.cta[0].n, -1), std::vector<int>(D.cta[0].m, -1)};
    for (int sd = 0; sd < 2; ++sd)
        for (int r = 0; r < mats[sd]->rows; ++r) row_at[sd][pos[sd][r]] = r;
    for (const ResCta& c : tab.cta) {
        if (c.slice0 != slices) return fail("slice tables are not contiguous", name, C);
        slices += c.ns_t + c.ns_a;
        if (c.n < T.rows || c.n > T.rows + 3 * C || c.m < A.rows || c.m > A.rows + 3 * C) return fail("sizes", name, C);
        if ((c.pos_t0 | c.pos_a0) & 3) return fail("a share does not start on 16 bytes", name, C);
        if (c.pos_t0 + ((c.own_t + 3) & ~3) > c.n || c.pos_a0 + ((c.own_a + 3) & ~3) > c.m) return fail("share past the end", name, C);
        for (int q = 0; q < c.ns_t + c.ns_a; ++q) {
            const ResSlice& e = tab.slices[c.slice0 + q];
            const int sd = q < c.ns_t ? 0 : 1, np = e.meta & 0xff, lg = (e.meta >> 8) & 0xf, nr = e.meta >> 12;
            if (e.pair0 < 0 || e.pair0 + np > c.pairs) return fail("slice outside its CTA's pairs", name, C);
            if (sd == 0 ? e.pair0 + np > c.pairs_t : e.pair0 < c.pairs_t) return fail("sides mixed", name, C);
            const int own = sd == 0 ? c.own_t : c.own_a, p0 = sd == 0 ? c.pos_t0 : c.pos_a0;
            if (e.own0 < 0 || e.own0 + nr > own || e.pos0 != p0 + e.own0) return fail("own range", name, C);
            for (int grp = 0; grp < nr; ++grp) {
                const int r = row_at[sd][e.pos0 + grp];
                ++got[sd][r];
                const Mat& M = *mats[sd];
                std::vector<float> prod;
                for (int p = M.ptr[r]; p < M.ptr[r + 1]; ++p) prod.push_back(M.val[p] * g[sd][M.idx[p]]);
                const float want = group_sum(prod, lg);
                const int G = 1 << lg;
                std::vector<float> acc(G, 0.0f);
                for (int l = 0; l < G; ++l)
                    for (int t = 0; t < np; ++t)
                        for (int h = 0; h < 2; ++h) {
                            const long long w = (c.pair0 + e.pair0 + t) * 64 + 2 * ((grp << lg) + l) + h;
                            const float x = idx[w] < 0 ? 0.0f : g[sd][row_at[1 - sd][idx[w]]];
                            acc[l] += val[w] * x;
                        }
                for (int o = G >> 1; o > 0; o >>= 1)
                    for (int l = 0; l + o < G; ++l) acc[l] += acc[l + o];
                if (std::memcmp(&acc[0], &want, 4) != 0) return fail("row sum", name, C);
            }
        }
    }
    for (auto& v : got)
        for (int k : v)
            if (k != 1) return fail("a row is summed by more or fewer than one slice", name, C);
    std::printf("ok %s C=%d slices=%d pairs=%lld\n", name.c_str(), C, slices, tab.pairs);
    return 0;
}

int main() {
    std::mt19937 rng(11);
    int bad = 0;
    struct Case { std::string name; int m, n, tmin, tmax, amin, amax; };
    const Case cases[] = {{"tiny", 1, 1, 1, 1, 1, 1},          {"small", 7, 33, 0, 4, 0, 9},
                          {"ragged", 700, 1753, 4, 12, 0, 31}, {"wide_rows", 90, 4000, 1, 6, 1, 1024},
                          {"long_columns", 3000, 60, 500, 1000, 1, 8}};
    for (const Case& c : cases) {
        const Mat T = random_mat(c.n, c.m, c.tmin, c.tmax, rng), A = random_mat(c.m, c.n, c.amin, c.amax, rng);
        for (int C = 1; C <= kResMaxCluster; C *= 2)
            for (bool by_block : {true, false}) bad |= check(c.name + (by_block ? "_f32" : "_f64"), T, A, by_block, C);
    }
    return bad;
}
