// Host-only checker of the row-block lists that the streaming kernels of a
// batch run when some of its instances iterate on chip (streamed_blocks,
// ganit_v2_b200/csrc/gb_problem.cuh), compiled and run by
// tests/test_stream_lists.py; no GPU involved.  FP32- and FP64-matrix kernels
// may run on schedules cut differently (the autotuner), and a block indexes the
// bitmaps of the schedule it was cut for: at each level the list's bitmap
// offsets have to give the row starts in the schedule of that level's view.
#include <cstdio>
#include <random>
#include <string>

#include "../ganit_v2_b200/csrc/gb_problem.cuh"

using namespace gb;

static int fail(const char* what, const std::string& where) {
    std::printf("FAIL %s: %s\n", where.c_str(), what);
    return 1;
}

static void put(DevSchedule& d, const Schedule& s) {
    d.nb = static_cast<int>(s.blocks.size());
    d.host_blocks = s.blocks;
    d.host_seg_block = s.seg_block;
}

// The window of block b in `bits` marks exactly the row starts of b.
static bool marks_rows(const Schedule& s, const int* ptr, RowBlock b) {
    const int off = b.slot_base, words = (4 * (((b.p1 + 3) >> 2) - (b.p0 >> 2)) + 31) / 32;
    if (off < 0 || off + words > static_cast<int>(s.bits.size())) return false;
    Schedule one;
    add_stream_bits(one, ptr, b);
    for (int w = 0; w < words; ++w)
        if (one.bits[w] != s.bits[off + w]) return false;
    return true;
}

template <class M, class V>
static int check(const Problem& P, const Schedule* a[2], const Schedule* t[2], const std::string& level) {
    constexpr int mw = sizeof(M) == 8;
    std::vector<RowBlock> l[2];
    streamed_blocks<M, V>(P, l[0], l[1]);
    for (int sd = 0; sd < 2; ++sd) {
        const DevMat& mat = sd == 0 ? P.A : P.AT;
        const Schedule& want = *(sd == 0 ? a : t)[mw];
        std::vector<int> seen(mat.rows, 0);
        for (const RowBlock& b : l[sd]) {
            if (P.res[sizeof(V) == 8].resident[b.inst]) return fail("an on-chip instance streams", level);
            if (b.kind == kStream && !marks_rows(want, mat.host_ptr.data(), b)) return fail("another schedule's bitmap", level);
            if (b.kind == kChunk && (b.slot_base + b.nchunks > want.nslots || b.counter >= want.ncounters))
                return fail("another schedule's slots", level);
            for (int r = b.r0; r < b.r1; ++r) seen[r] += b.kind == kChunk ? b.chunk == 0 : 1;
        }
        const std::vector<int>& off = sd == 0 ? P.row_off : P.col_off;
        for (int k = 0; k < P.count; ++k)
            for (int r = off[k]; r < off[k + 1]; ++r)
                if (seen[r] != (P.res[sizeof(V) == 8].resident[k] ? 0 : 1)) return fail("rows of the list", level);
    }
    std::printf("ok %s: %zu + %zu blocks\n", level.c_str(), l[0].size(), l[1].size());
    return 0;
}

int main() {
    std::mt19937 rng(3);
    Problem P;
    P.count = 4;
    P.row_off = {0, 300, 420, 1100, 1103};
    P.col_off = {0, 500, 700, 1500, 2500};
    P.A.rows = P.AT.cols = P.m = 1103;
    P.AT.rows = P.A.cols = P.n = 2500;
    for (DevMat* mat : {&P.A, &P.AT}) {
        mat->host_ptr.push_back(0);
        for (int r = 0; r < mat->rows; ++r)
            mat->host_ptr.push_back(mat->host_ptr.back() + (r == 1101 ? 9000 : r % 97 == 0 ? 700 : static_cast<int>(rng() % 14)));
    }
    auto cut = [&](const DevMat& mat, const std::vector<int>& off, int nnz, int rows) {
        const std::vector<int> b(P.count, nnz), r(P.count, rows);
        return build_schedule(mat.host_ptr.data(), off.data(), P.count, b.data(), r.data());
    };
    const Schedule a64 = cut(P.A, P.row_off, 2048, 256), t64 = cut(P.AT, P.col_off, 2048, 256);
    const Schedule a32 = cut(P.A, P.row_off, 1024, 64), t32 = cut(P.AT, P.col_off, 1024, 64);
    put(P.A.sched, a64);
    put(P.AT.sched, t64);
    for (ResPlan& R : P.res) R.resident = {0, 1, 0, 0};
    int bad = 0;
    for (bool tuned : {false, true}) {  // untuned: one schedule for all kernels
        if (tuned) {
            put(P.A.sched32, a32);
            put(P.AT.sched32, t32);
        }
        const Schedule *a[2] = {tuned ? &a32 : &a64, &a64}, *t[2] = {tuned ? &t32 : &t64, &t64};
        const std::string s = tuned ? "tuned " : "untuned ";
        bad |= check<float, float>(P, a, t, s + "f32/f32");
        bad |= check<float, double>(P, a, t, s + "f32/f64");
        bad |= check<double, double>(P, a, t, s + "f64/f64");
    }
    // the two cuts are told apart: FP64-matrix blocks do not pass for FP32-matrix ones
    std::vector<RowBlock> la, lt;
    streamed_blocks<double, double>(P, la, lt);
    bool all = true;
    for (const RowBlock& b : la) all &= b.kind != kStream || marks_rows(a32, P.A.host_ptr.data(), b);
    if (all) bad |= fail("the cuts do not differ", "test");
    return bad;
}
