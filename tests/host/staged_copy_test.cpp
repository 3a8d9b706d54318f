// CPU checks of efs_host::staged_copy: every byte arrives once and in place for
// sizes around chunk and ring edges, arrivals delayed; an exception of fetch or
// wait ends the copy and reaches the caller.  Prints "ok" or the first failure.
#include "efs_host.h"

#include <cstdio>
#include <stdexcept>

int main() {
    const size_t chunk = 1000;
    for (unsigned slots : {1u, 2u, 4u})
        for (unsigned T : {1u, 3u, 8u})
            for (size_t bytes : {(size_t)1, (size_t)999, (size_t)1000, (size_t)1001, (size_t)4000, (size_t)4001, (size_t)123457}) {
                std::vector<uint8_t> src(bytes), dst(bytes + 8, 0xEE);
                for (size_t i = 0; i < bytes; ++i) src[i] = (uint8_t)(i * 131 + i / 251);
                std::vector<std::vector<uint8_t>> ring(slots, std::vector<uint8_t>(chunk));
                std::vector<const uint8_t*> buf;
                for (auto& r : ring) buf.push_back(r.data());
                std::vector<size_t> started;
                size_t waited = 0;
                efs_host::staged_copy(dst.data(), bytes, buf.data(), slots, chunk, T,
                    [&](size_t c, size_t n) { started.push_back(n); (void)c; },
                    [&](size_t c) {          // the chunk arrives only now
                        std::memcpy(ring[c % slots].data(), src.data() + c * chunk, started[c]);
                        ++waited;
                    });
                bool ok = waited == (bytes + chunk - 1) / chunk && std::memcmp(dst.data(), src.data(), bytes) == 0;
                for (int i = 0; i < 8; ++i) ok = ok && dst[bytes + i] == 0xEE;
                if (!ok) { std::printf("FAIL slots %u T %u bytes %zu\n", slots, T, bytes); return 1; }
                for (int where = 0; where < 2; ++where) {
                    bool thrown = false;
                    try {
                        efs_host::staged_copy(dst.data(), bytes, buf.data(), slots, chunk, T,
                            [&](size_t c, size_t) { if (where == 0 && c >= (bytes + chunk - 1) / chunk / 2) throw std::runtime_error("x"); },
                            [&](size_t c) { if (where == 1 && c >= (bytes + chunk - 1) / chunk / 2) throw std::runtime_error("x"); });
                    } catch (const std::runtime_error&) { thrown = true; }
                    if (!thrown) { std::printf("FAIL no exception\n"); return 1; }
                }
            }
    std::printf("ok\n");
    return 0;
}
