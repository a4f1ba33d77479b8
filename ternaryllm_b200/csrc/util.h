// util.h -- error reporting shared by the host sources of libtllm.
#pragma once
#include <algorithm>
#include <cstdint>
#include <functional>
#include <system_error>
#include <thread>
#include <vector>

namespace tllm {

// Records a printf-style message for the calling thread (returned by tllm_last_error) and returns `code`.
int fail(int code, const char* fmt, ...);

// Runs `work` on this thread and on others, `most` and 32 in all at most; where the system gives no more threads, on fewer (an
// exception would leave through a C entry point).
template <typename F>
void on_threads(unsigned most, const F& work) {
    const unsigned n = std::max(1u, std::min({std::thread::hardware_concurrency(), 32u, most}));
    std::vector<std::thread> pool;
    pool.reserve(n);
    try {
        while (pool.size() + 1 < n) pool.emplace_back(std::cref(work));
    } catch (const std::system_error&) {
    }
    work();
    for (std::thread& th : pool) th.join();
}

// counts one kernel launch (tllm_launch_count)
void note_launch();

// decoders of the reference's formats into dense int8 [inners][columns]; return nullptr or a message
const char* decode_mcsc(const int32_t* row_idx, const int32_t* off, int columns, int inners, int tile_k,
                        std::vector<int8_t>* out);
const char* decode_cpu_format(int kind, int group, int chunk, const int32_t* meta, const void* ri, int ri32,
                              int64_t aux, int columns, int inners, std::vector<int8_t>* out);

}  // namespace tllm
