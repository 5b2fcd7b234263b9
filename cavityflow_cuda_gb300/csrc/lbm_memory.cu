// lbm_memory.cu -- device memory that a solver or a batch could do without: the
// second population arrays of the runs that take two steps a pass.  They are
// known here, so that an allocation of this library that finds no memory gets
// theirs: whoever needs the memory, they are the first to go.
#include "lbm_internal.h"

namespace lbm_detail {

namespace {

// Taken before a SecondArray's own mutex, never while one is held.
std::mutex list_mutex;
SecondArray* list = nullptr;

void release(SecondArray& a)
{
    const BesideCaptures beside;
    if (a.p || a.image) cudaDeviceSynchronize();  // queued passes still use them
    if (a.p) cudaFree(a.p);
    if (a.image) cudaFree(a.image);
    a.p = a.image = nullptr;
    a.bytes = 0;
}

}  // namespace

void add_second_array(SecondArray& a, int device)
{
    std::lock_guard<std::mutex> lock(list_mutex);
    a.device = device;
    a.listed = true;
    a.next = list;
    a.prev = nullptr;
    if (list) list->prev = &a;
    list = &a;
}

void remove_second_array(SecondArray& a)
{
    {
        std::lock_guard<std::mutex> lock(list_mutex);
        if (a.listed) {
            (a.prev ? a.prev->next : list) = a.next;
            if (a.next) a.next->prev = a.prev;
            a.listed = false;
        }
    }
    std::lock_guard<std::mutex> lock(a.mutex);
    release(a);
}

bool make_second_array(SecondArray& a, size_t bytes, size_t image_bytes)
{
    if (a.refused) return false;
    if (a.p) return true;
    const BesideCaptures beside;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess || bytes > free_b / 4 ||
        cudaMalloc(&a.p, bytes) != cudaSuccess ||
        (image_bytes > 0 && cudaMalloc(&a.image, image_bytes) != cudaSuccess)) {
        cudaGetLastError();
        release(a);
        a.refused = true;
        return false;
    }
    a.bytes = bytes + image_bytes;
    return true;
}

bool give_up_second_array(SecondArray& a)
{
    std::lock_guard<std::mutex> lock(a.mutex);
    a.refused = true;
    const bool held = a.p != nullptr;
    release(a);
    return held;
}

bool give_up_any_second_array(int device)
{
    std::lock_guard<std::mutex> lock(list_mutex);
    for (SecondArray* a = list; a; a = a->next) {
        if (a->device != device) continue;
        {
            std::lock_guard<std::mutex> own(a->mutex);
            if (!a->p) continue;
        }
        if (give_up_second_array(*a)) return true;
    }
    return false;
}

cudaError_t device_malloc(void** p, size_t bytes)
{
    cudaError_t e = cudaMalloc(p, bytes);
    int device = 0;
    while (e == cudaErrorMemoryAllocation && cudaGetDevice(&device) == cudaSuccess && give_up_any_second_array(device)) {
        cudaGetLastError();
        e = cudaMalloc(p, bytes);
    }
    return e;
}

}  // namespace lbm_detail
