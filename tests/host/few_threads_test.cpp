// CPU checks of efs_host::staged_copy where the host gives few threads or none:
// the address space is limited so that a thread's stack finds no room.  Every
// byte still arrives.  Prints "ok" or the first failure.
#include "efs_host.h"

#include <cstdio>
#include <cstdlib>
#include <stdexcept>
#include <sys/resource.h>

static size_t address_space() {
    size_t pages = 0;
    FILE* f = std::fopen("/proc/self/statm", "r");
    if (!f || std::fscanf(f, "%zu", &pages) != 1) std::exit(2);
    std::fclose(f);
    return pages * 4096;
}

int main() {
    const size_t chunk = 1000, bytes = 123457, slots = 4;
    std::vector<uint8_t> src(bytes), dst(bytes);
    for (size_t i = 0; i < bytes; ++i) src[i] = (uint8_t)(i * 131 + i / 251);
    std::vector<std::vector<uint8_t>> ring(slots, std::vector<uint8_t>(chunk));
    std::vector<const uint8_t*> buf;
    for (auto& r : ring) buf.push_back(r.data());
    for (size_t room : {(size_t)0, (size_t)2}) {                   // threads whose stacks fit
        const rlimit stack{8u << 20, RLIM_INFINITY};
        setrlimit(RLIMIT_STACK, &stack);                           // of new threads
        const size_t top = address_space() + (1u << 20) + room * (9u << 20);
        const rlimit lim{top, RLIM_INFINITY};
        if (setrlimit(RLIMIT_AS, &lim)) { std::printf("FAIL setrlimit\n"); return 1; }
        for (unsigned T : {1u, 8u}) {
            std::fill(dst.begin(), dst.end(), (uint8_t)0xEE);
            std::vector<size_t> started;
            started.reserve(bytes / chunk + 1);
            for (int fails : {0, 1}) {
                bool thrown = false;
                started.clear();
                try {
                    efs_host::staged_copy(dst.data(), bytes, buf.data(), slots, chunk, T,
                        [&](size_t c, size_t n) {
                            if (fails && c == 50) throw std::runtime_error("x");
                            started.push_back(n);
                        },
                        [&](size_t c) { std::memcpy(ring[c % slots].data(), src.data() + c * chunk, started[c]); });
                } catch (const std::runtime_error&) {
                    thrown = true;
                } catch (const std::exception& e) {
                    std::printf("FAIL room %zu T %u: %s\n", room, T, e.what());
                    return 1;
                }
                if (thrown != (fails == 1) || (!fails && std::memcmp(dst.data(), src.data(), bytes))) {
                    std::printf("FAIL room %zu T %u fails %d\n", room, T, fails);
                    return 1;
                }
            }
        }
        const rlimit open{RLIM_INFINITY, RLIM_INFINITY};
        setrlimit(RLIMIT_AS, &open);
    }
    std::printf("ok\n");
    return 0;
}
