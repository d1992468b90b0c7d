// host_pages.cpp -- host memory of large download arrays, on huge pages.
//
// A fresh array's pages are faulted in one by one by the copy into it, which
// costs more than the copy itself.  NumPy takes the functions below as the
// allocator of an array of 128 KB or more (its data memory handler, NEP 49), so the
// array owns its memory as any other; one of a huge page or more starts on a huge
// page and is faulted 2 MB at a time.
//
// A loop that downloads its results again and again drops the last ones when it
// has the next.  Through malloc their memory goes back to the kernel or not by
// what else lies at the heap's end, and the same run of ten boxes with sixty
// downloads took 196 ms in one process and 231 in another.  So blocks are mapped
// apart from the heap, and those freed last are kept for the next array of their
// size: of those on huge pages at most 512 MB, marked as free for the kernel to take
// when it needs them (MADV_FREE), of smaller ones 64 MB (there the mark costs 40 us
// an array, as much as the faults that it saves).  Any thread may free or allocate;
// one that finds the list in use goes without.
#include <sys/mman.h>

#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>

namespace {

constexpr size_t kHugePage = size_t(1) << 21, kPage = 4096;
constexpr size_t kMapped = size_t(1) << 17, kGrain = size_t(1) << 16;   // smallest block mapped; sizes below a huge page

// Ahead of every block.
struct alignas(16) Header {
    size_t size;       // bytes asked for
    size_t mapped;     // bytes of the block's pages, 0: from malloc
};

Header* header_of(void* p) { return static_cast<Header*>(p) - 1; }

void unmap_block(void* data, size_t mapped) { munmap(static_cast<char*>(data) - kPage, mapped + kPage); }

// Freed blocks, the last one at the end.
struct Kept {
    struct {
        void* data;
        size_t mapped;
    } block[256];
    int count = 0;
    size_t bytes = 0;
    const size_t most;
    const bool give_back;   // mark the pages as free for the kernel
    std::mutex mutex;

    Kept(size_t limit, bool give) : most(limit), give_back(give) {}

    // A block of exactly `mapped` bytes, the last one freed, or null.
    void* take(size_t mapped)
    {
        const std::unique_lock<std::mutex> lock(mutex, std::try_to_lock);
        if (!lock.owns_lock()) return nullptr;
        for (int i = count - 1; i >= 0; --i) {
            if (block[i].mapped != mapped) continue;
            void* p = block[i].data;
            drop(i, 1);
            return p;
        }
        return nullptr;
    }

    // Keeps a block, in the place of those kept longest where there is no room.
    bool keep(void* data, size_t mapped)
    {
        if (mapped > most) return false;
        const std::unique_lock<std::mutex> lock(mutex, std::try_to_lock);
        if (!lock.owns_lock()) return false;
        int out = 0;
        for (size_t left = bytes; count - out == 256 || left + mapped > most; ++out) {
            left -= block[out].mapped;
            unmap_block(block[out].data, block[out].mapped);
        }
        drop(0, out);
        if (give_back) madvise(data, mapped, MADV_FREE);
        block[count].data = data;
        block[count++].mapped = mapped;
        bytes += mapped;
        return true;
    }

private:
    void drop(int at, int n)
    {
        for (int k = at; k < at + n; ++k) bytes -= block[k].mapped;
        for (int k = at + n; k < count; ++k) block[k - n] = block[k];
        count -= n;
    }
};

// (never destroyed: arrays may be freed after the library's own end)
Kept& kept_of(size_t size)
{
    static Kept* const huge = new Kept(size_t(512) << 20, true);
    static Kept* const small = new Kept(size_t(64) << 20, false);
    return size < kHugePage ? *small : *huge;
}

// `mapped` bytes from the returned address on, a huge page's where there is one,
// and a page for the header ahead of them.
void* map_block(size_t size, size_t mapped)
{
    const size_t align = size < kHugePage ? kPage : kHugePage, room = mapped + align + kPage;
    char* base = static_cast<char*>(mmap(nullptr, room, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    if (base == MAP_FAILED) return nullptr;
    const uintptr_t at = reinterpret_cast<uintptr_t>(base);
    char* data = base + ((at + kPage + align - 1) / align * align - at);
    const size_t ahead = static_cast<size_t>(data - kPage - base), behind = room - ahead - kPage - mapped;
    if (ahead) munmap(base, ahead);
    if (behind) munmap(data + mapped, behind);
    // (the last huge page where the array fills half of it; refused: ordinary pages)
    if (size >= kHugePage) madvise(data, (size + kHugePage / 2) / kHugePage * kHugePage, MADV_HUGEPAGE);
    return data;
}

void* pages_malloc(void*, size_t size)
{
    if (size > SIZE_MAX / 2) return nullptr;
    void* data = nullptr;
    size_t mapped = 0;
    if (size < kMapped) {
        Header* h = static_cast<Header*>(std::malloc(size + sizeof(Header)));
        data = h ? h + 1 : nullptr;
    } else {
        const size_t grain = size < kHugePage ? kGrain : kHugePage;
        mapped = (size + grain - 1) / grain * grain;
        data = kept_of(size).take(mapped);
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
    const Header h = *header_of(p);
    if (!h.mapped) std::free(header_of(p));
    else if (!kept_of(h.size).keep(p, h.mapped)) unmap_block(p, h.mapped);
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
