// plan_tests -- tests of the context's host side (buffers, graph keys, plans of
// launches) without a GPU: device-memory calls go to a fake, nothing is launched.
#include <functional>
#include <iostream>
#include <stdexcept>

#include "cmc_capi_internal.hpp"

using namespace cmc;

namespace {

int g_checks = 0;

void require(bool ok, const char* what) {
    ++g_checks;
    if (!ok) throw std::runtime_error(what);
}

// A device whose free memory is one run of bytes from kBase on: an allocation
// takes the lowest address where it fits.
struct FakeDevice {
    static constexpr uintptr_t kBase = 1 << 20;
    size_t size = 0;
    std::map<uintptr_t, size_t> live;
    uint32_t allocs = 0, releases = 0;
} g_device;

cudaError_t fake_alloc(void** out, size_t n) {
    ++g_device.allocs;
    uintptr_t at = FakeDevice::kBase;
    for (auto& [p, m] : g_device.live) {
        if (p - at >= n) break;
        at = p + m;
    }
    if (at + n > FakeDevice::kBase + g_device.size) return cudaErrorMemoryAllocation;
    g_device.live[at] = n;
    *out = reinterpret_cast<void*>(at);
    return cudaSuccess;
}

cudaError_t fake_release(void* p) {
    ++g_device.releases;
    return g_device.live.erase(reinterpret_cast<uintptr_t>(p)) ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t fake_available(size_t* n) {
    *n = g_device.size;
    for (auto& [p, m] : g_device.live) *n -= m;
    return cudaSuccess;
}

void use_fake(Ctx& c, size_t bytes) {
    g_device = FakeDevice{};
    g_device.size = bytes;
    c.memory = DeviceMemory{fake_alloc, fake_release, fake_available};
    c.sms = 148;
    c.smem_optin = 232448;
}

int grow_pool(Ctx& c, size_t bytes) {
    void* p = c.d_slots;
    const int rc = c.grow_bytes(p, c.slots_cap, bytes, 1, "pool");
    c.d_slots = static_cast<char*>(p);
    return rc;
}

// A buffer that cannot grow stays as it is, unless giving it up makes the room.
void check_grow() {
    Ctx c;
    use_fake(c, 1000);
    require(grow_pool(c, 400) == CMC_OK && c.slots_cap == 400, "first allocation");
    char* const first = c.d_slots;
    require(grow_pool(c, 300) == CMC_OK && g_device.allocs == 1, "a smaller need allocates nothing");
    require(grow_pool(c, 5000) == CMC_ENOMEM, "more than the device has");
    require(c.d_slots == first && c.slots_cap == 400 && g_device.live.size() == 1 && g_device.releases == 0,
            "a failed allocation leaves the buffer");
    require(grow_pool(c, 800) == CMC_OK && c.slots_cap == 800 && g_device.live.size() == 1,
            "the old buffer makes room for the new one");
    c.fixed_memory = true;  // a stream capture
    const uint32_t calls = g_device.allocs + g_device.releases;
    char* const kept = c.d_slots;
    require(grow_pool(c, 900) == CMC_ENOMEM && g_device.allocs + g_device.releases == calls && c.d_slots == kept &&
                c.slots_cap == 800,
            "no allocation or release during a capture");
    c.fixed_memory = false;
}

// A graph is replayed only with the buffers, and the sizes, it was captured with.
void check_graphs() {
    Ctx c;
    use_fake(c, 1000);
    std::vector<Job> jobs(1);
    cmc_params p;
    require(cmc_derive_params(CMC_MODE_BGH25, 64, 16, 3, 96, 100, 1, &p) == CMC_OK &&
                c.make_job(p, 0, 1000, 0, jobs[0]) == CMC_OK,
            "a job");
    const std::vector<uint32_t> bounds{0, 1};
    auto replays = [&]() {
        for (const Ctx::GraphEntry& g : c.graphs)
            if (g.key == c.graph_key(jobs, bounds, 1000, 1000)) return true;
        return false;
    };
    require(grow_pool(c, 800) == CMC_OK, "pool");
    const uintptr_t large = reinterpret_cast<uintptr_t>(c.d_slots);
    c.graphs.push_back(Ctx::GraphEntry{c.graph_key(jobs, bounds, 1000, 1000)});
    require(replays(), "the same call");
    // a call whose pool does not fit, then the smaller one it falls back to: at
    // no point may the graph of the larger pool match a smaller one at its address
    require(grow_pool(c, 2000) == CMC_ENOMEM, "too large a pool");
    require(!replays() || c.slots_cap >= 800, "a graph replays in its own pool");
    require(grow_pool(c, 100) == CMC_OK, "the pool of the fallback");
    require(!replays() || (reinterpret_cast<uintptr_t>(c.d_slots) == large && c.slots_cap >= 800),
            "a graph replays in its own pool, also after a fallback");
    require(grow_pool(c, 900) == CMC_OK && c.graphs.empty(), "graphs go with the buffer they name");

    // every pointer counts in full
    for (void** at : {(void**)&c.d_jobs, (void**)&c.d_bits, (void**)&c.d_out, (void**)&c.d_slots,
                      (void**)&c.d_job_failed, (void**)&c.h_failed}) {
        void* const was = *at;
        *at = reinterpret_cast<void*>(0x7ffffffffff0);
        const std::string a = c.graph_key(jobs, bounds, 0xfffffffe, 0xfffffffe);
        *at = reinterpret_cast<void*>(0x7ffffffffff1);
        require(a != c.graph_key(jobs, bounds, 0xfffffffe, 0xfffffffe), "a pointer is part of the key");
        *at = was;
    }
}

}  // namespace

int main() {
    const std::pair<const char*, void (*)()> tests[] = {{"buffers", check_grow}, {"graphs", check_graphs}};
    int bad = 0;
    for (auto& [name, test] : tests) {
        try {
            test();
        } catch (const std::exception& e) {
            std::cerr << "FAILED " << name << ": " << e.what() << '\n';
            ++bad;
        }
    }
    if (!bad) std::cout << "ALL PLAN TESTS PASSED (" << g_checks << " checks)\n";
    return bad != 0;
}
