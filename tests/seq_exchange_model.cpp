/* The exchanges of a sequential pass (csrc/seq_exchange.h) on modelled
 * mbarriers: CL CTAs of NT threads in step, one thread of one CTA giving up at
 * one exchange.  Prints the largest transaction count in bytes any barrier held
 * and how many threads gave up.  argv: CTA, thread and exchange of the one that
 * gives up, and the exchanges in all. */
#include <algorithm>
#include <cstdio>
#include <cstdlib>

#include "../mset_b200/csrc/seq_exchange.h"

constexpr int CL = 16, NT = 32;
constexpr long BYTES = 32768;  // an exchange's share of one CTA at 256 x 256
struct Barrier {
    int pending = 1;
    long tx = 0;
    unsigned phase = 0;
    void settle() {
        if (pending == 0 && tx == 0) {
            ++phase;
            pending = 1;
        }
    }
};

int main(int argc, char **argv) {
    if (argc != 5) return 2;
    const int bad_cta = atoi(argv[1]), bad_thread = atoi(argv[2]), bad_at = atoi(argv[3]), total = atoi(argv[4]);
    Barrier bar[CL][2];
    mset::SeqProgress at[CL][NT];
    long worst = 0;
    auto arm = [&](int q, int w) {
        bar[q][w].pending -= 1;
        bar[q][w].tx += BYTES;
        bar[q][w].settle();
    };
    auto push = [&](int q, int w, long bytes) {
        bar[q][w].tx -= bytes;
        bar[q][w].settle();
        worst = std::max(worst, std::labs(bar[q][w].tx));
    };
    for (int q = 0; q < CL; ++q)
        for (int w = 0; w < 2; ++w) arm(q, w);
    for (int e = 0; e < total; ++e) {
        const int w = e & 1;  // rows, then columns, in turn; what is pushed goes to the other
        if (e > 0)
            for (int q = 0; q < CL; ++q)
                for (int t = 0; t < NT; ++t) {
                    mset::SeqProgress &x = at[q][t];
                    bool done = true;
                    if (x.waits())
                        done = bar[q][w].phase > x.ph[w] && !(q == bad_cta && t == bad_thread && e == bad_at);
                    x.waited(w, done);
                    if (t == 0 && x.arms()) arm(q, w);
                }
        // a row task's columns belong to all CTAs, a column task's rows to one
        for (int q = 0; q < CL; ++q)
            for (int t = 0; t < NT; ++t) {
                if (!at[q][t].sends()) continue;
                if (w == 0)
                    for (int p = 0; p < CL; ++p) push(p, 1, BYTES / CL / NT);
                else push(t % CL, 0, BYTES / NT);
            }
    }
    int dead = 0;
    for (auto &c : at)
        for (auto &x : c) dead += x.dead;
    printf("%ld %d\n", worst, dead);
    return 0;
}
