// CPU check of efs_host::parallel_chunks where the host gives few threads or
// none: the address space is limited so that a thread's stack finds no room.
// Every item is still visited once, by the chunk it belongs to.  Prints "ok".
#include "efs_host.h"

#include <cstdio>
#include <cstdlib>
#include <sys/resource.h>

int main() {
    const size_t n = 1000003;
    const unsigned T = 16;
    std::vector<uint8_t> seen(n);
    const rlimit stack{8u << 20, RLIM_INFINITY};
    setrlimit(RLIMIT_STACK, &stack);                               // of new threads
    for (size_t room : {(size_t)0, (size_t)3, (size_t)100}) {      // threads whose stacks fit
        std::fill(seen.begin(), seen.end(), (uint8_t)0);
        size_t pages = 0;
        FILE* f = std::fopen("/proc/self/statm", "r");
        if (!f || std::fscanf(f, "%zu", &pages) != 1) return 2;
        std::fclose(f);
        const rlimit lim{pages * 4096 + (1u << 20) + room * (9u << 20), RLIM_INFINITY};
        if (setrlimit(RLIMIT_AS, &lim)) return 2;
        efs_host::parallel_chunks(n, T, [&](unsigned t, size_t lo, size_t hi) {
            for (size_t i = lo; i < hi; ++i) seen[i] += (uint8_t)(1 + t);
        });
        const rlimit open{RLIM_INFINITY, RLIM_INFINITY};
        setrlimit(RLIMIT_AS, &open);
        for (unsigned t = 0; t < T; ++t)
            for (size_t i = n * t / T; i < n * (t + 1) / T; ++i)
                if (seen[i] != 1 + t) { std::printf("FAIL room %zu item %zu\n", room, i); return 1; }
    }
    std::printf("ok\n");
    return 0;
}
