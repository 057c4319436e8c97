// Randomised host simulation of the tcgen05 GEMM's mbarrier protocol as the kernel runs it, over the functions of
// elanfmt_gb300/csrc/ewf_umma.h that it uses; compiled with g++ by tests/test_umma_ring_cpu.py.  One CTA: a TMA
// producer per operand, the MMA issuer and eight epilogue warps over `tiles` tiles of `nk` k-stages in a ring of
// 4 to 16 slots, every role testing its next slot early; copies land in any order, MMA commits complete in issue
// order, all interleaved at random.  An mbarrier is its completed-phase count n, the arrivals and the copies its phase
// still expects; a wait with parity P passes when n % 2 != P.
// Checked: the run ends; a slot is refilled only after the stage before in it was consumed; the issuer reads a stage
// exactly when both operands have landed, and writes an accumulator only after it was drained; an
// epilogue warp reads a tile exactly when its MMAs are complete.  In half of the runs waits give up at random, as when
// a limit runs out (the flag they raise makes later ones give up): the roles then still end, each after
// its own copies and MMAs, within the polls of bounded_drain.
// Prints "ok <runs>" or the first failure.
#include <cstdio>
#include <deque>
#include <random>
#include <vector>

#include "ewf_umma.h"

using namespace ewf_umma;

struct Bar {
    int n = 0, arrived = 0, need = 1, tx = 0;
    void settle()
    {
        if (arrived == need && tx == 0) {
            arrived = 0;
            ++n;
        }
    }
    void arrive(int expect = 0)
    {
        tx += expect;
        ++arrived;
        settle();
    }
    void land()
    {
        --tx;
        settle();
    }
    bool pass(uint32_t parity) const { return (uint32_t)(n & 1) != parity; }
};

constexpr int WARPS = 8;
constexpr int POLLS = 3000;  // of a drain (in the kernel DRAIN_POLLS)

struct Sim {
    int tiles, nk, ns;
    bool failing, err = false;
    std::mt19937 rng;
    std::vector<Bar> full, empty;
    Bar acc_full[2], acc_empty[2];
    std::vector<int> consumed, landed[2];             // per slot: stages consumed, copies of each operand landed
    std::vector<std::pair<int, int>> flying;          // (operand, slot) of the copies on their way
    std::deque<std::pair<int, int>> commits;          // (0 empty / 1 acc_full, slot or buffer), in issue order
    int boxes[2], drained[2] = {0, 0}, computed[2] = {0, 0};
    const char *bad = nullptr;

    struct Producer {
        int op, q = 0, s = 0;
        uint32_t parity = 1;
        bool ready = true, done = false, drained = false;
        int at = -1, polls = 0;  // the stage whose copy it drains, and the polls so far
    } prod[2];
    struct Issuer {
        int i = 0, kt = 0, s = 0, g = 0;
        uint32_t parity = 0;
        bool ready = false, open = false, done = false;
    } mma;
    int epi[WARPS] = {};

    // a wait that has not passed: whether it gives up
    bool gives_up()
    {
        if (failing && (err || rng() % 40 == 0)) err = true;
        return err;
    }

    Sim(int tiles_, int nk_, int ns_, bool failing_, unsigned seed) : tiles(tiles_), nk(nk_), ns(ns_), failing(failing_), rng(seed), full(ns_), empty(ns_), consumed(ns_, 0)
    {
        for (auto &b : full) b.need = 2;
        for (auto &b : acc_empty) b.need = WARPS;
        for (int op = 0; op < 2; ++op) {
            landed[op].assign(ns, 0);
            prod[op].op = op;
            boxes[op] = 1 + (int)(rng() % 2);  // a transposed operand comes in several boxes
        }
    }

    bool produce(Producer &p)
    {
        if (p.done) return last_copies(p);
        if (!p.ready && !empty[p.s].pass(p.parity)) {
            p.done = gives_up();
            return p.done;
        }
        int s1;
        uint32_t p1;
        ring_next(p.s, p.parity, ns, &s1, &p1);
        const bool next = empty[s1].pass(p1);
        if (consumed[p.s] != p.q / ns) bad = "a slot is refilled while in use";
        full[p.s].arrive(boxes[p.op]);
        for (int b = 0; b < boxes[p.op]; ++b) flying.push_back({p.op, p.s});
        p.ready = next;
        p.s = s1;
        p.parity = p1;
        if (++p.q == tiles * nk) p.done = true;
        return true;
    }
    // the kernel's loop over the last ns stages, bounded_drain on each, a poll at a time
    bool last_copies(Producer &p)
    {
        if (p.drained) return false;
        if (p.at < 0) p.at = p.q > ns ? p.q - ns : 0;
        if (p.at == p.q) {
            p.drained = true;
            for (const auto &c : flying)
                if (c.first == p.op) bad = "a producer ends before its copies landed";
            return true;
        }
        if (full[ring_slot(p.at, ns)].pass(ring_full_parity(p.at, ns)) || ++p.polls == POLLS) {
            ++p.at;
            p.polls = 0;
        }
        return true;
    }
    bool issue()
    {
        Issuer &m = mma;
        if (m.done) return false;
        if (!m.open) {
            const int b = acc_buf(m.i);
            if (acc_needs_free(m.i) && !acc_empty[b].pass(acc_free_parity(m.i))) {
                m.done = gives_up();
                return m.done;
            }
            if (!err && drained[b] != m.i / 2) bad = "an accumulator is written before it was drained";
            m.open = true;
        }
        if (!m.ready && !full[m.s].pass(m.parity)) {
            m.done = gives_up();
            return m.done;
        }
        int s1;
        uint32_t p1;
        ring_next(m.s, m.parity, ns, &s1, &p1);
        const bool next = full[s1].pass(p1);
        for (int op = 0; op < 2; ++op)
            if (landed[op][m.s] != (m.g / ns + 1) * boxes[op]) bad = "a stage is read before, or after a refill of, its copies";
        commits.push_back({0, m.s});
        m.ready = next;
        m.s = s1;
        m.parity = p1;
        ++m.g;
        if (++m.kt == nk) {
            commits.push_back({1, acc_buf(m.i)});
            m.kt = 0;
            m.open = false;
            if (++m.i == tiles) m.done = true;
        }
        return true;
    }
    bool drain(int w)
    {
        const int i = epi[w], b = acc_buf(i);
        if (i == tiles) return false;
        const bool got = acc_full[b].pass(acc_full_parity(i));
        if (!got && !gives_up()) return false;
        if (!err && computed[b] != i / 2 + 1) bad = "an accumulator is read before its MMAs completed";
        ++epi[w];
        const int before = acc_empty[b].n;
        acc_empty[b].arrive();
        if (acc_empty[b].n != before) ++drained[b];
        return true;
    }
    bool land()
    {
        if (flying.empty()) return false;
        const size_t q = rng() % flying.size();
        const auto c = flying[q];
        flying.erase(flying.begin() + q);
        ++landed[c.first][c.second];
        full[c.second].land();
        return true;
    }
    bool complete()
    {
        if (commits.empty()) return false;
        const auto c = commits.front();
        commits.pop_front();
        if (c.first == 0) {
            ++consumed[c.second];
            empty[c.second].arrive();
        } else {
            ++computed[c.second];
            acc_full[c.second].arrive();
        }
        return true;
    }
    bool ended() const
    {
        for (int w = 0; w < WARPS; ++w)
            if (epi[w] != tiles) return false;
        return prod[0].drained && prod[1].drained && mma.done && flying.empty() && commits.empty();
    }
    const char *run()
    {
        // the roles' speeds differ from run to run, so that each is at times the one that is waited for
        const int speed[5] = {1 + (int)(rng() % 6), 1 + (int)(rng() % 6), 1 + (int)(rng() % 6), 1 + (int)(rng() % 6), 1 + (int)(rng() % 6)};
        const int sum = speed[0] + speed[1] + speed[2] + speed[3] + speed[4];
        for (long idle = 0; !bad && !ended();) {
            int who = (int)(rng() % sum), r = 0;
            while (who >= speed[r]) who -= speed[r++];
            const bool moved = r == 0 ? produce(prod[rng() % 2]) : r == 1 ? issue() : r == 2 ? drain((int)(rng() % WARPS)) : r == 3 ? land() : complete();
            idle = moved ? 0 : idle + 1;
            if (idle > 100000) return "deadlock";
        }
        return bad;
    }
};

int main()
{
    int runs = 0;
    unsigned seed = 1;
    for (int rep = 0; rep < 2; ++rep)
    for (int ns = 4; ns <= 16; ++ns)
        for (int tiles = 1; tiles <= 5; ++tiles)
            for (int nk : {1, 2, 3, 4, 5, 8, 15, 16, 17, 33}) {
                const bool failing = seed & 1;
                const char *e = Sim(tiles, nk, ns, failing, seed++).run();
                if (e) {
                    printf("FAIL %s: slots %d tiles %d nk %d seed %u\n", e, ns, tiles, nk, seed - 1);
                    return 1;
                }
                ++runs;
            }
    printf("ok %d\n", runs);
    return 0;
}
