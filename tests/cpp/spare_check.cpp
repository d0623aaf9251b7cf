// Allocations that fail: what a context keeps for speed alone is given back and
// the allocation tried again.  The device is a counter here (cudaMalloc and
// cudaFree below), so nothing but the host logic of internal.h runs.
#include <cstdio>
#include <cstdlib>
#include <map>

#include "../../streamsim_gb300/csrc/internal.h"

#define CHECK(c)                                                                \
    do {                                                                        \
        if (!(c)) {                                                             \
            std::fprintf(stderr, "check failed: %s (line %d)\n", #c, __LINE__); \
            std::exit(1);                                                       \
        }                                                                       \
    } while (0)

namespace {
constexpr size_t kDevice = size_t(100) << 20;
std::map<void*, size_t> held;
size_t used = 0;
}  // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n)
{
    if (used + n > kDevice) return cudaErrorMemoryAllocation;
    *p = std::malloc(1);
    held[*p] = n;
    used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p)
{
    if (!p) return cudaSuccess;
    CHECK(held.count(p) == 1);  // once each
    used -= held[p];
    held.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

namespace facetcu {
void ColumnPlan::release()
{
    for (DeviceBuffer* b : {&shares, &groups, &meta, &words, &partial}) b->release();
    state = kUnknown;
}
}  // namespace facetcu

using namespace facetcu;

struct Context final : Spare {
    Workspace ws;
    RasterBuffers raster;
    ColumnPlan plan;
    int asked = 0;
    bool give_back() override
    {
        ++asked;
        bool any = ws.kept != 0;
        ws.drop_blocks();
        any |= plan.give_back();
        any |= raster.give_back();
        return any;
    }
};

bool refused(DeviceBuffer& b, size_t n)
{
    try {
        b.reserve(n);
    } catch (const Error& e) {
        CHECK(e.code == FACETCU_OUT_OF_MEMORY);
        CHECK(b.ptr == nullptr && b.bytes == 0);
        return true;
    }
    return false;
}

int main()
{
    constexpr size_t MB = size_t(1) << 20;
    {
        Context c;
        DeviceBuffer want;
        { ScratchBuffer s(c.ws); s.reserve(50 * MB); }
        CHECK(c.ws.kept == 50 * MB && used == 50 * MB);
        CHECK(refused(want, 80 * MB));  // no context: as any allocation
        CHECK(c.asked == 0 && c.ws.kept == 50 * MB);
        const SpareScope scope(&c);
        CHECK(!refused(want, 80 * MB));  // kept scratch
        CHECK(c.asked == 1 && c.ws.kept == 0 && used == 80 * MB);
        CHECK(refused(want, 120 * MB));  // more than there is: refused, nothing held
        CHECK(c.asked == 2 && used == 0);
        // lent scratch stays
        ScratchBuffer lent(c.ws);
        lent.reserve(30 * MB);
        { ScratchBuffer s(c.ws); s.reserve(40 * MB); }
        CHECK(!refused(want, 70 * MB) && used == 100 * MB);
        want.release();
        // scratch itself asks too
        c.plan.words.reserve(60 * MB);
        c.plan.state = ColumnPlan::kMade;
        ScratchBuffer more(c.ws);
        CHECK(more.reserve(50 * MB) != nullptr);
        CHECK(c.plan.state == ColumnPlan::kUnknown && used == 80 * MB);
    }
    CHECK(used == 0);
    {
        Context c;
        const SpareScope scope(&c);
        DeviceBuffer want;
        // a plan that is being made stays, and so do lists in use
        c.plan.words.reserve(40 * MB);
        c.raster.heads.reserve(30 * MB);
        {
            const RasterUse use(c.raster);
            CHECK(refused(want, 60 * MB) && used == 70 * MB);
        }
        CHECK(!refused(want, 60 * MB) && used == 100 * MB);  // the lists went
        CHECK(c.plan.words.ptr && !c.raster.heads.ptr);
        {
            Context other;  // a nested call of another context, then this one again
            const SpareScope inner(&other);
            want.release();
            CHECK(refused(want, 80 * MB) && other.asked == 1);
        }
        const int before = c.asked;
        CHECK(refused(want, 80 * MB) && c.asked == before + 1);
    }
    CHECK(used == 0);
    std::printf("spare memory ok\n");
    return 0;
}
