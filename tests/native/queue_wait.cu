// A wait of the tile queue that runs out (a tile whose first steps nothing takes), and
// an engine that finds its error word set.  Built and run by test_gpu_queue_error.py;
// exits 0 and prints "ok" if every check holds.
#include <cstdio>
#include <fstream>
#include <sstream>
#include <string>
#include <vector>

#include "sbe_engine.h"
#include "sbe_queue.cuh"

using namespace sbe;

// items of 2 chunks of `ntiles` tiles; the chunks before counter's start are never taken
__global__ void drain(TileQueue q, int *prog, int *ran, int polls)
{
    for (int item = next_item(q); item >= 0; item = next_item(q)) {
        const int tile = item % q.ntiles, s0 = item / q.ntiles * q.chunk;
        if (!tile_ready(q, prog + tile, s0, s0 == 0, polls)) continue;
        if (threadIdx.x == 0) atomicAdd(ran, 1);
        tile_done(q, prog + tile, s0 + q.chunk);
    }
}

static int failures = 0;
static void check(bool ok, const char *what)
{
    if (!ok) {
        std::printf("failed: %s\n", what);
        ++failures;
    }
}
template <class F> static bool throws(F f)
{
    try {
        f();
    } catch (const CudaError &) {
        return true;
    }
    return false;
}

int main(int argc, char **argv)
{
    const int ntiles = 40, chunk = 64, nctas = 16;
    int *d = nullptr;   // queue counters, error word, run items, progress
    if (cudaMalloc(&d, sizeof(int) * (4 + ntiles)) != cudaSuccess) return 2;
    for (int first : {0, 3}) {   // the counter starts past `first` tiles: their second chunk waits in vain
        std::vector<int> h(4 + ntiles, 0);
        h[0] = first;
        cudaMemcpy(d, h.data(), sizeof(int) * h.size(), cudaMemcpyHostToDevice);
        drain<<<nctas, 32>>>(TileQueue{d, d + 2, ntiles, chunk, 2 * ntiles}, d + 4, d + 3, 1 << 20);
        check(cudaDeviceSynchronize() == cudaSuccess, "the launch ends");
        cudaMemcpy(h.data(), d, sizeof(int) * h.size(), cudaMemcpyDeviceToHost);
        check(h[0] == 0 && h[1] == 0, "the counters are put back");
        check(h[2] == (first > 0), "the error word");
        check(first > 0 ? h[3] <= 2 * ntiles - 2 * first : h[3] == 2 * ntiles, "items run");
        for (int t = 0; t < first; ++t) check(h[4 + t] == 0, "a tile whose wait ran out is left alone");
    }

    // the host side: every reader of an engine's results sees the word
    std::ifstream in(argc > 1 ? argv[1] : "");
    std::stringstream text;
    text << in.rdbuf();
    const auto root = parse_cfg(text.str());
    std::string unsupported;
    const Problem p = problem_from_cfg(*root, &unsupported);
    cudaStream_t st;
    cudaStreamCreate(&st);
    {
        Engine e(0, st, 128, 1);
        EngineOptions eo;
        const int id = e.add(p, eo);
        while (e.max_remaining_ticks() > 0) e.step();
        std::vector<double> j, band(4), occ((size_t)p.nshots() * p.Nk[0]);
        double cp[NSLOT];
        e.raw_outputs(id, j, cp);
        e.harmonics(id, 0.0855, 4, band.data());
        check(e.snapshots(id, occ.data(), nullptr, nullptr) == p.nshots(), "snapshots");
        const int one = 1;
        cudaMemcpy(e.queue_error(), &one, sizeof(one), cudaMemcpyHostToDevice);
        check(throws([&] { e.harmonics(id, 0.0855, 4, band.data()); }), "harmonics see the error");
        check(throws([&] { e.snapshots(id, occ.data(), nullptr, nullptr); }), "snapshots see the error");
        check(throws([&] { e.fetch_async(id); e.raw_outputs(id, j, cp); }), "outputs see the error");
    }
    cudaStreamDestroy(st);
    cudaFree(d);
    if (failures == 0) std::printf("ok\n");
    return failures == 0 ? 0 : 1;
}
