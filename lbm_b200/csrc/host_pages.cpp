// host_pages.cpp -- host memory of large download arrays, on huge pages.
//
// A fresh array's pages are faulted in one by one by the copy into it, which
// costs more than the copy itself.  NumPy takes the functions below as the
// allocator of an array (its data memory handler, NEP 49), so the array owns its
// memory as any other; one of a huge page or more starts on a huge page and is
// faulted 2 MB at a time.
//
// A loop that downloads its results again and again drops the last ones when it
// has the next.  Through malloc their memory goes back to the kernel or not by
// what else lies at the heap's end, and the same run of ten boxes with sixty
// downloads took 196 ms in one process and 231 in another.  So blocks are mapped
// apart from the heap, and a few that were freed are kept for the next array of
// their size: at most 512 MB and 256 blocks, their pages marked as free for the
// kernel to take when it needs them (MADV_FREE).  Any thread may free or allocate;
// one that finds the list in use goes without.
#include <sys/mman.h>

#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace {

constexpr size_t kHugePage = size_t(1) << 21, kPage = 4096;
constexpr size_t kKeptBytes = size_t(512) << 20;
constexpr int kKeptBlocks = 256;

// Ahead of every block.
struct alignas(16) Header {
    size_t size;       // bytes asked for
    size_t mapped;     // bytes of the block's huge pages, 0: from malloc
};

Header* header_of(void* p) { return static_cast<Header*>(p) - 1; }

struct Kept {
    void* data;
    size_t mapped;
};
Kept g_kept[kKeptBlocks];
int g_kept_count = 0;
size_t g_kept_bytes = 0;
std::mutex g_kept_mutex;

// A kept block of exactly `mapped` bytes, the last one freed, or null.
void* take_kept(size_t mapped)
{
    const std::unique_lock<std::mutex> lock(g_kept_mutex, std::try_to_lock);
    if (!lock.owns_lock()) return nullptr;
    for (int i = g_kept_count - 1; i >= 0; --i) {
        if (g_kept[i].mapped != mapped) continue;
        void* p = g_kept[i].data;
        for (int k = i + 1; k < g_kept_count; ++k) g_kept[k - 1] = g_kept[k];
        --g_kept_count;
        g_kept_bytes -= mapped;
        return p;
    }
    return nullptr;
}

bool keep(void* data, size_t mapped)
{
    const std::unique_lock<std::mutex> lock(g_kept_mutex, std::try_to_lock);
    if (!lock.owns_lock() || g_kept_count == kKeptBlocks || mapped > kKeptBytes - g_kept_bytes) return false;
    madvise(data, mapped, MADV_FREE);
    g_kept[g_kept_count++] = {data, mapped};
    g_kept_bytes += mapped;
    return true;
}

// Whole huge pages that start at the returned address, a page for the header
// ahead of them.
void* map_block(size_t size, size_t mapped)
{
    const size_t room = mapped + kHugePage + kPage;
    char* base = static_cast<char*>(mmap(nullptr, room, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    if (base == MAP_FAILED) return nullptr;
    const uintptr_t at = reinterpret_cast<uintptr_t>(base);
    char* data = base + ((at + kPage + kHugePage - 1) / kHugePage * kHugePage - at);
    const size_t ahead = static_cast<size_t>(data - kPage - base), behind = room - ahead - kPage - mapped;
    if (ahead) munmap(base, ahead);
    if (behind) munmap(data + mapped, behind);
    // (the last huge page where the array fills half of it; refused: ordinary pages)
    madvise(data, (size + kHugePage / 2) / kHugePage * kHugePage, MADV_HUGEPAGE);
    return data;
}

void* pages_malloc(void*, size_t size)
{
    if (size > SIZE_MAX / 2) return nullptr;
    void* data = nullptr;
    size_t mapped = 0;
    if (size < kHugePage) {
        Header* h = static_cast<Header*>(std::malloc(size + sizeof(Header)));
        data = h ? h + 1 : nullptr;
    } else {
        mapped = (size + kHugePage - 1) / kHugePage * kHugePage;
        data = take_kept(mapped);
        if (!data) data = map_block(size, mapped);
    }
    if (data) *header_of(data) = {size, mapped};
    return data;
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
    if (!p) return;
    const size_t mapped = header_of(p)->mapped;
    if (!mapped) std::free(header_of(p));
    else if (!keep(p, mapped)) munmap(static_cast<char*>(p) - kPage, mapped + kPage);
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
