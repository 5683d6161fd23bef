// Calls of CUDASimulation that only C++ can make, one per argument; prints
// "ok" or what went wrong (run by test_host_calls_gpu.py).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "flamegpu/flamegpu.h"

using flamegpu::CUDASimulation;
using flamegpu::ModelDescription;

namespace {

int fails = 0;
void expect(bool ok, const char* what, long long value) {
    if (ok) return;
    std::printf("%s (%lld)\n", what, value);
    ++fails;
}

ModelDescription& model() {
    static ModelDescription m("host_calls");
    static bool made = false;
    if (!made) {
        flamegpu::AgentDescription a = m.newAgent("agent");
        a.newVariable<int>("x");
        a.newVariable<int>("y");
        made = true;
    }
    return m;
}

// columns of n rows in page-locked memory
struct Rows {
    uint32_t n;
    uint32_t* id;
    int *x, *y;
    Rows(uint32_t rows, int first) : n(rows) {
        cudaMallocHost(&id, 4ull * n);
        cudaMallocHost(&x, 4ull * n);
        cudaMallocHost(&y, 4ull * n);
        for (uint32_t i = 0; i < n; ++i) {
            id[i] = i + 1;
            x[i] = first + static_cast<int>(i);
            y[i] = -x[i];
        }
    }
    ~Rows() {
        for (void* p : {static_cast<void*>(id), static_cast<void*>(x), static_cast<void*>(y)}) cudaFreeHost(p);
    }
    std::vector<std::pair<std::string, const void*>> in() const { return {{"_id", id}, {"x", x}, {"y", y}}; }
    std::vector<std::pair<std::string, void*>> out() { return {{"_id", id}, {"x", x}, {"y", y}}; }
};

// A refused population of a count that is no multiple of four leaves the one that was there.
void unset_id() {
    for (uint32_t n : {1u, 5u, 1021u, 32'767u, 32'769u, 100'003u}) {
        CUDASimulation sim(model());
        Rows first(n + 2, 10), second(n, 5000), got(n + 2, 0);
        sim.setPopulationColumns("agent", "default", n + 2, first.in());
        second.id[n == 32'769u ? n - 1 : n / 2] = 0;  // once in the last, partial piece
        bool refused = false;
        try {
            sim.setPopulationColumns("agent", "default", n, second.in());
        } catch (const flamegpu::exception::InvalidArgument&) {
            refused = true;
        }
        expect(refused, "an unset id was taken, n", n);
        expect(sim.getPopulationColumns("agent", "default", got.out(), n + 2) == n + 2, "the population is lost, n", n);
        for (uint32_t i = 0; i < n + 2 && !fails; ++i)
            expect(got.id[i] == first.id[i] && got.x[i] == first.x[i] && got.y[i] == first.y[i], "changed row", i);
    }
}

// The list's own columns as sources: copied in the order given.
void own_columns() {
    for (uint32_t n : {5u, 100'003u}) {
        CUDASimulation sim(model());
        Rows rows(n, 10), got(n, 0);
        sim.setPopulationColumns("agent", "default", n, rows.in());
        const void* x = sim.getDeviceVariable("agent", "x");
        const void* y = sim.getDeviceVariable("agent", "y");
        const void* id = sim.getDeviceVariable("agent", "_id");
        sim.setPopulationDevice("agent", "default", n, {{"x", y}, {"y", x}, {"_id", id}}, n + 1);
        sim.getPopulationColumns("agent", "default", got.out(), n);
        for (uint32_t i = 0; i < n && !fails; ++i)  // x became y, then y took the new x
            expect(got.id[i] == rows.id[i] && got.x[i] == rows.y[i] && got.y[i] == rows.y[i], "row", i);
    }
}

}  // namespace

int main(int argc, char** argv) {
    const std::string which = argc > 1 ? argv[1] : "";
    if (which == "unset_id") unset_id();
    else if (which == "own_columns") own_columns();
    else return 2;
    if (!fails) std::printf("ok\n");
    return fails ? 1 : 0;
}
