// Runs a stack's maps, then writes one pair's fault word into its record as the column pass that gave
// up waiting would have left it, and collects: prints a line per case, "1" for results, "0: message".
#include <cuda_runtime.h>

#include <array>
#include <cmath>
#include <cstdio>
#include <deque>
#include <map>
#include <string>
#include <utility>
#include <vector>

#define private public
#include "engine.hpp"

int main() {
    constexpr int n = 4, w = 64, h = 48;
    std::vector<std::vector<float>> img(n, std::vector<float>(w * h));
    const float* p[n];
    int ws[n], hs[n];
    for (int k = 0; k < n; ++k) {
        for (int i = 0; i < w * h; ++i) {
            const int x = i % w + k, y = i / w - k;
            img[k][i] = (float)(std::sin(0.31 * x) * std::cos(0.17 * y) + 0.3 * std::sin(0.05 * x * y));
        }
        p[k] = img[k].data(), ws[k] = w, hs[k] = h;
    }
    zc::Engine e(0);
    zc_shift_result out[n - 1];
    if (!e.stack_load(n, p, ws, hs, nullptr, true, false, 0)) return std::printf("load: %s\n", e.err.c_str()), 1;
    auto collect = [&](int pair, size_t at, unsigned v, int dft) {
        e.err.clear();
        if (e.stack_enqueue() < 0 || cudaDeviceSynchronize() != cudaSuccess) return false;
        for (int k = 0; k < n - 1; ++k)  // a map without the tensor-core stage leaves its word as it was
            if (cudaMemset(e.stack_res_.as<char>() + k * zc::kMapRecord + 28, 0, 4) != cudaSuccess) return false;
        if (pair >= 0 && cudaMemcpy(e.stack_res_.as<char>() + pair * zc::kMapRecord + at, &v, 4, cudaMemcpyHostToDevice) != cudaSuccess)
            return false;
        e.dft_pieces_ = dft;  // read by the collection only: the maps above ran without the stage
        const bool ok = e.stack_collect(out);
        e.dft_pieces_ = 0;
        std::printf(ok ? "1\n" : "0: %s\n", e.err.c_str());
        return true;
    };
    for (int pair = -1; pair < n - 1; ++pair)
        if (!collect(pair, 24, 1, 0)) return 1;
    if (!collect(1, 28, 1, 1) || !collect(-1, 0, 0, 1) || !collect(-1, 0, 0, 0)) return 1;
    return 0;
}
