// Host-only checker of the exchange between the CTAs of a cluster
// (cluster_exchange, ganit_v2_b200/csrc/gb_resident.cuh), compiled and run by
// tests/test_exchange.py; no GPU involved.  A model of the mbarriers runs the
// halves of several iterations on the shares that res_deal gives, with every
// message delayed at random: no message of one iteration may reach a barrier
// whose phase belongs to another, and every CTA gets to the end.  The same
// model without the shares of CTAs that own nothing finds the overtaking that
// they prevent.
#include <cstdio>
#include <random>
#include <string>
#include <vector>

#include "../ganit_v2_b200/csrc/gb_resident.cuh"

using namespace gb;

struct Bar {
    int pending = 1;   // the CTA's own arrival
    long long tx = 0;  // bytes announced and not yet in
    int phase = 0;
    void settle() {
        if (pending == 0 && tx == 0) {
            pending = 1;
            ++phase;
        }
    }
};
struct Message {
    int to, half;
    long long bytes;
};

// Whether a run of `iters` iterations went wrong: 1 overtaking, 2 no end.
static int run(const std::vector<ResCta>& cta, int iters, bool shares, std::mt19937& rng) {
    const int C = static_cast<int>(cta.size());
    auto own = [&](int c, int side) { return side == 0 ? cta[c].own_t : cta[c].own_a; };
    // `shares`: CTAs that own nothing take part too
    auto bytes = [&](int c, int side) { return shares || own(c, side) ? static_cast<long long>(share_bytes<float>(own(c, side))) : 0; };
    const long long total[2] = {share_total<float>(cta[0].n, shares ? cta[0].idle_t : 0),
                                share_total<float>(cta[0].m, shares ? cta[0].idle_a : 0)};
    std::vector<std::array<Bar, 2>> bar(C);
    std::vector<int> half(C, 0), sent(C, 0);  // half c is in; whether it has sent
    std::vector<Message> air;
    auto done = [&] {
        for (int h : half)
            if (h < 2 * iters) return false;
        return true;
    };
    const int slow = static_cast<int>(rng() % C);  // messages to this CTA take longest
    for (long long step = 0; !done(); ++step) {
        if (step > 200000) return 2;
        const bool deliver = !air.empty() && rng() % 3 != 0;
        if (deliver) {
            const size_t k = rng() % air.size();
            const Message msg = air[k];
            if (msg.to == slow && rng() % 64 != 0) continue;
            Bar& b = bar[msg.to][msg.half & 1];
            if (b.phase != msg.half >> 1) return 1;
            b.tx -= msg.bytes;
            b.settle();
            air[k] = air.back();
            air.pop_back();
            continue;
        }
        const int c = static_cast<int>(rng() % C);
        if (half[c] == 2 * iters) continue;
        const int side = half[c] & 1;
        Bar& b = bar[c][side];
        if (!sent[c]) {
            sent[c] = 1;
            b.tx += total[side] - bytes(c, side);
            --b.pending;
            for (int p = 0; p < C; ++p)
                if (p != c && bytes(c, side)) air.push_back({p, half[c], bytes(c, side)});
            b.settle();
        }
        if (b.phase > half[c] >> 1) {
            ++half[c];
            sent[c] = 0;
        }
    }
    return 0;
}

int main() {
    std::mt19937 rng(17);
    struct Case {
        const char* name;
        std::vector<int> rows, cols;  // lengths of the rows of A and of A^T
        int C;
    };
    auto ragged = [&](int k, int lo, int hi) {
        std::vector<int> v(k);
        for (int& x : v) x = lo + static_cast<int>(rng() % (hi - lo + 1));
        return v;
    };
    const Case cases[] = {{"ten_rows", ragged(10, 700, 1000), ragged(5000, 0, 4), 16},
                          {"one_row", {1000}, ragged(2000, 0, 1), 8},
                          {"seven_rows", {1024, 5, 1, 33, 32, 31, 65}, ragged(1500, 0, 3), 8},
                          {"eleven_columns", ragged(6000, 1, 2), ragged(11, 700, 1000), 16},
                          {"both_few", ragged(3, 2, 9), ragged(9, 0, 3), 4},
                          {"every_cta_owns", ragged(800, 3, 30), ragged(2000, 2, 9), 8}};
    int bad = 0;
    for (const Case& c : cases) {
        std::array<ResHist, 2> H;
        const std::vector<int>* lens[2] = {&c.cols, &c.rows};
        for (int sd = 0; sd < 2; ++sd) {
            std::vector<int> ptr{0};
            for (int l : *lens[sd]) ptr.push_back(ptr.back() + l);
            if (!res_hist_rows(ptr.data(), 0, static_cast<int>(lens[sd]->size()), -1, H[sd])) return 1;
            H[sd].count();
        }
        ResDeal D;
        res_deal(H, c.C, D);
        int idle[2] = {0, 0};
        for (const ResCta& k : D.cta) {
            idle[0] += k.own_t == 0;
            idle[1] += k.own_a == 0;
        }
        for (const ResCta& k : D.cta)
            if (k.idle_t != idle[0] || k.idle_a != idle[1]) {
                std::printf("FAIL %s: idle CTAs miscounted\n", c.name);
                return 1;
            }
        int wrong = 0, without = 0;
        for (int k = 0; k < 300; ++k) {
            wrong += run(D.cta, 5, true, rng) != 0;
            without += run(D.cta, 5, false, rng) != 0;
        }
        if (wrong || (without > 0) != (idle[0] + idle[1] > 0)) {
            std::printf("FAIL %s: %d of 300 runs overtaken, %d without the idle CTAs' shares\n", c.name, wrong, without);
            bad = 1;
        } else {
            std::printf("ok %s: C=%d, %d + %d own nothing, overtaken without their shares in %d of 300 runs\n", c.name, c.C,
                        idle[0], idle[1], without);
        }
    }
    return bad;
}
