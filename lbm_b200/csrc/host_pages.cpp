// host_pages.cpp -- host memory of large download arrays, on huge pages.
//
// A fresh array's pages are faulted in one by one by the copy into it, which
// costs more than the copy itself.  An allocation that starts on a huge page
// and asks for huge pages is faulted 2 MB at a time.  NumPy takes the functions
// as the allocator of an array (its data memory handler, NEP 49), so the array
// owns its memory as any other.  The memory is malloc's: a block of a huge page
// or more is the part of a larger one that starts on a huge page (aligned
// allocations are found again less often: 207 instead of 196 ms for a run of ten
// boxes with sixty downloads).
#include <sys/mman.h>

#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>

namespace {

constexpr size_t kHugePage = size_t(1) << 21, kPage = 4096;

// Ahead of every block.
struct alignas(16) Header {
    void* base;      // malloc's pointer
    size_t size;
};

Header* header_of(void* p) { return static_cast<Header*>(p) - 1; }

void* place(void* base, size_t offset, size_t size)
{
    Header* h = reinterpret_cast<Header*>(static_cast<char*>(base) + offset);
    h->base = base;
    h->size = size;
    return h + 1;
}

void* pages_malloc(void*, size_t size)
{
    const size_t room = sizeof(Header) + (size < kHugePage ? 0 : kHugePage);
    if (size > SIZE_MAX - room) return nullptr;
    void* base = std::malloc(size + room);
    if (!base || size < kHugePage) return base ? place(base, 0, size) : nullptr;
    const uintptr_t at = reinterpret_cast<uintptr_t>(base), first = (at + kPage - 1) / kPage * kPage;
    madvise(reinterpret_cast<void*>(first), at + size + room - first, MADV_HUGEPAGE);   // (refused: ordinary pages)
    const uintptr_t data = (at + sizeof(Header) + kHugePage - 1) / kHugePage * kHugePage;
    return place(base, data - sizeof(Header) - at, size);
}

void* pages_calloc(void* ctx, size_t n, size_t size)
{
    if (size && n > SIZE_MAX / size) return nullptr;
    void* p = pages_malloc(ctx, n * size);
    if (p) std::memset(p, 0, n * size);
    return p;
}

void pages_free(void*, void* p, size_t)
{
    if (p) std::free(header_of(p)->base);
}

void* pages_realloc(void* ctx, void* p, size_t size)
{
    void* q = pages_malloc(ctx, size);
    if (!q || !p) return q;
    const size_t kept = header_of(p)->size;
    std::memcpy(q, p, kept < size ? kept : size);
    pages_free(ctx, p, kept);
    return q;
}

// NumPy's PyDataMem_Handler, version 1.
struct DataMemHandler {
    char name[127];
    unsigned char version;
    void* ctx;
    void* (*malloc)(void*, size_t);
    void* (*calloc)(void*, size_t, size_t);
    void* (*realloc)(void*, void*, size_t);
    void (*free)(void*, void*, size_t);
};

// (lives as long as the library: arrays may outlive whatever refers to it)
const DataMemHandler kHostPages = {"lbm_b200_pages", 1, nullptr, pages_malloc, pages_calloc, pages_realloc, pages_free};

}  // namespace

extern "C" const void* lbm_host_pages(void) { return &kHostPages; }
