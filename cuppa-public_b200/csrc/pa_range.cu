// pa_range.cu -- see pa_range.h.  Pages of device memory mapped side by side into one
// reserved span of addresses, so that a piece may cover any run of them.
#include "pa_range.h"

#include <cuda.h>

#include <algorithm>

#include "pa_internal.h"

namespace pa {
namespace {

// Pages of 64 MB, smaller ones below 8 GB, where a page can still be free between two
// results (a page takes the driver some 0.2 ms to map: 0.4 GB in 2 MB pages 45 ms); and
// addresses for kSpan times the range: regroup() maps pages at unused ones.
constexpr uint64_t kPage = 64ull << 20, kPagesLeast = 128;
constexpr uint64_t kSpan = 16;

// Driver entry points, fetched through the runtime so the library needs no link
// against libcuda.
struct Driver {
    decltype(&cuMemGetAllocationGranularity) granularity = nullptr;
    decltype(&cuMemAddressReserve) reserve = nullptr;
    decltype(&cuMemAddressFree) unreserve = nullptr;
    decltype(&cuMemCreate) create = nullptr;
    decltype(&cuMemRelease) release = nullptr;
    decltype(&cuMemMap) map = nullptr;
    decltype(&cuMemUnmap) unmap = nullptr;
    decltype(&cuMemSetAccess) access = nullptr;
    bool ok = false;

    template <typename F>
    static bool fetch(const char *name, F *f)
    {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) != cudaSuccess) {
            (void)cudaGetLastError();
            return false;
        }
        *f = reinterpret_cast<F>(p);
        return q == cudaDriverEntryPointSuccess && p;
    }
    Driver()
    {
        ok = fetch("cuMemGetAllocationGranularity", &granularity) &&
             fetch("cuMemAddressReserve", &reserve) && fetch("cuMemAddressFree", &unreserve) &&
             fetch("cuMemCreate", &create) && fetch("cuMemRelease", &release) &&
             fetch("cuMemMap", &map) && fetch("cuMemUnmap", &unmap) &&
             fetch("cuMemSetAccess", &access);
    }
};

const Driver &driver()
{
    static const Driver d;
    return d;
}

CUmemAllocationProp page_prop(int device)
{
    CUmemAllocationProp prop = {};
    prop.type = CU_MEM_ALLOCATION_TYPE_PINNED;
    prop.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
    prop.location.id = device;
    return prop;
}

bool set_access(CUdeviceptr p, uint64_t bytes, int device)
{
    CUmemAccessDesc a = {};
    a.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
    a.location.id = device;
    a.flags = CU_MEM_ACCESS_FLAGS_PROT_READWRITE;
    return driver().access(p, bytes, &a, 1) == CUDA_SUCCESS;
}

}  // namespace

bool DeviceRange::open(int device, uint64_t bytes)
{
    const Driver &drv = driver();
    if (base_ || !drv.ok || bytes == 0) return false;
    const CUmemAllocationProp prop = page_prop(device);
    size_t least = 0;
    if (drv.granularity(&least, &prop, CU_MEM_ALLOC_GRANULARITY_MINIMUM) != CUDA_SUCCESS || !least)
        return false;
    device_ = device;
    page_ = std::min(kPage, std::max<uint64_t>(bytes / kPagesLeast, 1));
    page_ = (page_ + least - 1) / least * least;
    const uint64_t count = bytes / page_;
    CUdeviceptr base = 0;
    if (count == 0 || drv.reserve(&base, kSpan * count * page_, 0, 0, 0) != CUDA_SUCCESS) return false;
    base_ = reinterpret_cast<unsigned char *>(base);
    pages_.assign(kSpan * count, 0);
    bool ok = true;
    for (uint64_t i = 0; ok && i < count; ++i) {
        CUmemGenericAllocationHandle h = 0;
        ok = drv.create(&h, page_, &prop, 0) == CUDA_SUCCESS;
        if (!ok) break;
        ok = drv.map(base + i * page_, page_, 0, h, 0) == CUDA_SUCCESS;
        if (ok) pages_[i] = h;
        else drv.release(h);
    }
    ok = ok && set_access(base, count * page_, device);
    if (!ok) {
        close();
        return false;
    }
    arena_.add(0, count * page_);
    return true;
}

void DeviceRange::close()
{
    if (!base_) return;
    const Driver &drv = driver();
    const CUdeviceptr base = reinterpret_cast<CUdeviceptr>(base_);
    for (uint64_t i = 0; i < pages_.size(); ++i)
        if (pages_[i]) {
            drv.unmap(base + i * page_, page_);
            drv.release(pages_[i]);
        }
    drv.unreserve(base, page_ * pages_.size());
    base_ = nullptr;
    pages_.clear();
    arena_.clear();
}

void *DeviceRange::regroup(uint64_t bytes)
{
    if (!base_) return nullptr;
    if (void *p = take(bytes)) return p;
    const Driver &drv = driver();
    const CUdeviceptr base = reinterpret_cast<CUdeviceptr>(base_);
    const uint64_t want = (bytes + page_ - 1) / page_;
    if (want == 0 || want > pages_.size()) return nullptr;
    // whole pages inside free pieces
    std::vector<uint64_t> from;
    for (const auto &f : arena_.pieces()) {
        const uint64_t lo = (f.first + page_ - 1) / page_, hi = (f.first + f.second) / page_;
        for (uint64_t i = lo; i < hi && from.size() < want; ++i) from.push_back(i);
    }
    if (from.size() < want) return nullptr;
    // the first run of unused addresses
    uint64_t to = 0, run = 0;
    for (uint64_t i = 0; i < pages_.size() && run < want; ++i) run = pages_[i] ? 0 : (to = i + 1, run + 1);
    if (run < want) return nullptr;
    to -= want;
    for (uint64_t k = 0; k < want; ++k) {
        const uint64_t i = from[k];
        arena_.cut(i * page_, page_);
        // a page that can't be moved is lost to the range, and given back to the device
        const bool out = drv.unmap(base + i * page_, page_) == CUDA_SUCCESS;
        if (!out) return nullptr;
        const CUmemGenericAllocationHandle h = pages_[i];
        pages_[i] = 0;
        if (drv.map(base + (to + k) * page_, page_, 0, h, 0) != CUDA_SUCCESS) {
            drv.release(h);
            return nullptr;
        }
        pages_[to + k] = h;
        if (!set_access(base + (to + k) * page_, page_, device_)) return nullptr;
        arena_.add((to + k) * page_, page_);
    }
    return take(bytes);
}

}  // namespace pa
