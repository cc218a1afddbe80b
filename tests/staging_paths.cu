// Drives the host <-> device copies of fm_staging.cu on a CPU, linked against fake_cuda.cpp in
// place of the CUDA runtime.  Prints one line per scenario.
#include "../fumeng_b200/csrc/fm_staging.cu"

#include <sys/mman.h>

#include <cstdio>

#include "fake_cuda.h"

namespace {

constexpr size_t kMiB = size_t(1) << 20;

// Sends `kinds.size()` arrays of `bytes` in and back, the last one's result added as doubles,
// and prints what happened.
void round_trip(const char* name, size_t bytes, const std::vector<cudaMemoryType>& kinds)
{
    fm_ctx ctx;
    g_direct = g_staged = 0;
    g_ranges.clear();
    const size_t n = bytes / sizeof(double);
    std::vector<std::vector<double>> host, dev, back;
    for (size_t k = 0; k < kinds.size(); ++k) {
        host.emplace_back(n);
        for (size_t i = 0; i < n; ++i) host[k][i] = (double)(i * 7 + k);
        dev.emplace_back(n, -1.0);
        back.emplace_back(n, 100.0);
        if (kinds[k] != cudaMemoryTypeUnregistered) {
            g_ranges.push_back(Range{reinterpret_cast<char*>(host[k].data()), bytes, kinds[k]});
            g_ranges.push_back(Range{reinterpret_cast<char*>(back[k].data()), bytes, kinds[k]});
        }
    }
    std::vector<fm::InCopy> in;
    std::vector<fm::OutCopy> out;
    for (size_t k = 0; k < kinds.size(); ++k) {
        in.push_back(fm::InCopy{dev[k].data(), host[k].data(), bytes});
        out.push_back(fm::OutCopy{back[k].data(), dev[k].data(), bytes, k + 1 == kinds.size()});
    }
    const cudaError_t e1 = fm::copy_in(&ctx, nullptr, in);
    const int in_direct = g_direct, in_staged = g_staged;
    g_direct = g_staged = 0;
    const cudaError_t e2 = e1 == cudaSuccess ? fm::copy_results(&ctx, nullptr, out) : e1;
    bool same = true;
    for (size_t k = 0; k < kinds.size(); ++k)
        for (size_t i = 0; i < n; ++i)
            same = same && back[k][i] == host[k][i] + (k + 1 == kinds.size() ? 100.0 : 0.0);
    std::printf("%s %d %d %s %d %d %d %d\n", name, (int)e1, (int)e2, same ? "same" : "different", in_direct, in_staged > 0,
                g_direct, g_staged > 0);
    std::fflush(stdout);
    fm::staging_release(&ctx);
}

}  // namespace

int main()
{
    const cudaMemoryType page = cudaMemoryTypeUnregistered, locked = cudaMemoryTypeHost, managed = cudaMemoryTypeManaged;
    round_trip("small", kMiB, {page, page});
    round_trip("pageable", 20 * kMiB, {page, page});
    round_trip("locked", 20 * kMiB, {locked, locked, page});
    round_trip("locked_small_rest", 7 * kMiB, {locked, managed, page});
    for (int threads : {0, 2}) {
        g_threads_left = threads;
        round_trip(threads == 0 ? "no_threads" : "two_threads", 20 * kMiB, {page, page});
    }
    g_threads_left = 1 << 30;
    g_no_pinned = true;
    round_trip("no_ring", 20 * kMiB, {page, locked, page});
    g_no_pinned = false;
    {
        // memory of a device where host memory belongs: an error, and the host never touches it
        fm_ctx ctx;
        const size_t bytes = 20 * kMiB;
        char* wall = static_cast<char*>(mmap(nullptr, bytes, PROT_NONE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
        std::vector<char> dev(bytes);
        g_ranges.assign(1, Range{wall, bytes, cudaMemoryTypeDevice});
        const cudaError_t e1 = fm::copy_in(&ctx, nullptr, {fm::InCopy{dev.data(), wall, bytes}});
        const cudaError_t e2 = fm::copy_results(&ctx, nullptr, {fm::OutCopy{wall, dev.data(), bytes}});
        std::printf("device %d %d\n", (int)e1, (int)e2);
        fm::staging_release(&ctx);
    }
    return 0;
}
