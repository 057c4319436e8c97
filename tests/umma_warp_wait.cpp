// Host model of the tcgen05 GEMM's bounded wait (warp_wait of elanfmt_gb300/csrc/ewf_umma.h, which the kernel
// uses), compiled with g++ by tests/test_umma_ring_cpu.py.  The lanes of a warp are threads and the warp's vote a
// barrier between them; a barrier phase that completes is seen by each lane from a poll of its own on, at
// random around the limit, and another wait's failure likewise.  Checked: every lane gets the same answer, also
// where lanes deciding by themselves would not.  Prints "ok <runs> <runs where lanes alone would have parted>".
#include <barrier>
#include <cstdio>
#include <random>
#include <thread>
#include <vector>

#include "ewf_umma.h"

constexpr int LANES = 8;

int main()
{
    std::mt19937 rng(5);
    int runs = 0, parted = 0;
    for (int limit : {0, 1, 2, 5, 1023, 1024, 1030, 2060})
        for (int rep = 0; rep < 12; ++rep) {
            int seen[LANES], fails[LANES];
            for (int l = 0; l < LANES; ++l) {
                seen[l] = limit + (int)(rng() % 3) - 1;                              // first poll that passes
                fails[l] = rep % 3 == 2 ? 1022 + (int)(rng() % 3) : 1 << 30;         // poll from which the failure flag is seen
            }
            bool held[2] = {true, true}, got[LANES];
            std::barrier sync(LANES);
            std::vector<std::thread> warp;
            for (int l = 0; l < LANES; ++l)
                warp.emplace_back([&, l] {
                    int polls = 0, votes = 0;
                    auto vote = [&](bool x) {  // all lanes', as __all_sync
                        bool &h = held[votes & 1];
                        if (!x) __atomic_store_n(&h, false, __ATOMIC_RELAXED);
                        sync.arrive_and_wait();
                        const bool all = __atomic_load_n(&h, __ATOMIC_RELAXED);
                        sync.arrive_and_wait();
                        if (l == 0) h = true;
                        ++votes;
                        return all;
                    };
                    got[l] = ewf_umma::warp_wait(limit, [&] { return polls++ >= seen[l]; }, [&] { return polls > fails[l]; }, vote);
                });
            for (auto &t : warp) t.join();
            bool alone[LANES];
            for (int l = 0; l < LANES; ++l) {
                int polls = 0;
                alone[l] = ewf_umma::warp_wait(limit, [&] { return polls++ >= seen[l]; }, [&] { return polls > fails[l]; }, [](bool x) { return x; });
            }
            bool split = false;
            for (int l = 1; l < LANES; ++l) {
                split = split || alone[l] != alone[0];
                if (got[l] != got[0]) {
                    printf("FAIL lanes parted: limit %d rep %d\n", limit, rep);
                    return 1;
                }
            }
            parted += split;
            ++runs;
        }
    if (!parted) {
        printf("FAIL no run puts the lanes' own answers apart\n");
        return 1;
    }
    printf("ok %d %d\n", runs, parted);
    return 0;
}
