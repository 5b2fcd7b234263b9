// lbm_internal.h -- definitions shared by the C ABI translation units
// (lbm_capi.cu, lbm_batch.cu); not part of the public interface.
#pragma once

#include <atomic>
#include <cstdint>
#include <exception>
#include <mutex>
#include <new>
#include <cuda_runtime.h>

#include "../../include/lbm_gb300.h"
#include "lbm_kernels.h"

struct lbm_batch;

namespace lbm_detail {

// Device buffer in which the getters pack a call's values for one contiguous
// copy to the host; `idle` is recorded behind the copy that last used it.
struct PackBuffer {
    std::mutex mutex;
    cudaEvent_t idle = nullptr;
    void* p = nullptr;
    size_t bytes = 0;
    bool owned = true;  // false: the end of the solver's macros array
};
void free_pack(PackBuffer& b);

// Lets this thread allocate and free while a stream is captured elsewhere in
// global mode, which such calls would otherwise break.  For memory that a call
// could do without: the calls that take it worked beside a capture when they
// took none.
class BesideCaptures {
public:
    BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    ~BesideCaptures() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    BesideCaptures(const BesideCaptures&) = delete;
    BesideCaptures& operator=(const BesideCaptures&) = delete;

private:
    cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

// The second population array of a solver's or a batch's runs that take two steps
// a pass, and the batch plan's image.  The owner could do without: it is made
// only while it takes at most a quarter of the free memory, and given up, for
// good, when an allocation of this library on that device finds too little
// (lbm_memory.cu).
struct SecondArray {
    std::mutex mutex;  // held to use or change what follows, and by a run until its launches are queued
    void* p = nullptr;
    void* image = nullptr;
    std::atomic<size_t> bytes{0};  // of both; read without the mutex, so that nobody waits for a run to know it
    bool refused = false;      // no memory for it, or given up
    int device = 0;
    bool listed = false;
    SecondArray* prev = nullptr;
    SecondArray* next = nullptr;
};
void add_second_array(SecondArray& a, int device);
void remove_second_array(SecondArray& a);                            // frees it too
bool make_second_array(SecondArray& a, size_t bytes, size_t image_bytes);  // a.mutex held; whether it is there
bool give_up_second_array(SecondArray& a);                           // whether there was one
bool give_up_any_second_array(int device);
// cudaMalloc on the current device that gives second arrays up rather than fail.
// The caller holds no SecondArray's mutex.
cudaError_t device_malloc(void** p, size_t bytes);
template <class T>
cudaError_t device_malloc(T** p, size_t bytes)
{
    return device_malloc(reinterpret_cast<void**>(p), bytes);
}

// The error flag of a batch's kernels, which step all domains.  The device word
// is cleared by the first domain that finds it set; `count` is how often that
// happened, and every domain reports each time once (lbm_solver::faults_seen).
struct BatchFault {
    std::mutex mutex;
    int* word = nullptr;
    std::atomic<uint64_t> count{0};
};

}  // namespace lbm_detail

struct lbm_solver {
    lbm::Grid g{};
    int storage = 0;
    int device = 0;
    lbm::Params p{};
    int bc[6] = {0, 0, 0, 0, 0, 0};
    void* dd = nullptr;             // populations, 19 * g.S elements
    uint8_t* flags = nullptr;       // one byte per cell, reference layout
    void* macros = nullptr;         // 4 * cells values (rho, jx, jy, jz)
    bool macros_fresh = false;
    bool macros_checked = true;     // the error flag that came with them has been looked at
    double* scratch = nullptr;      // reduction partials (4 per block) + result (4)
    unsigned long long* counts = nullptr;  // cavity-flag check counters [0..1], kernel error flag [2],
                                           // work words of the pair kernel [3], step words [4] (see step_words)
    double* host_out = nullptr;     // pinned: the reduction's 4 doubles, then the error flag of compute_macros
    float* staging = nullptr;       // 16-bit storage: one packed slot cuboid
    size_t staging_elems = 0;
    int64_t counter = 0;
    bool last_alpha = false;
    int lid_y = -1;                 // fast path: lid row (ny) or 0 for none; -1: flag-array path
    int variant = 0;                // launch variant of the vectorised kernels
    bool fma = false;               // FP64: fused multiply-adds in the vectorised steps
    int lid_mode = 0;               // LBM_LID_INJECTION or LBM_LID_MOVING_WALL; the wall moves
                                    // while p.wall_y > 0
    lbm_detail::PackBuffer pack;    // the getters' packing buffer
    lbm_detail::PackBuffer* batch_pack = nullptr;  // a batch domain's: shared by the batch
    lbm_detail::SecondArray second; // lbm_run's second population array (ensure_pairs)
    bool pairs = true;              // lbm_run may take two steps a pass: no launch variant was asked for
    cudaStream_t capture_stream = nullptr;
    cudaGraphExec_t graph = nullptr;
    int64_t device_bytes = 0;
    bool owns_dd = true;            // false: populations live in a batch's pool
    lbm_batch* batch = nullptr;     // the batch this solver is a domain view of
    lbm_detail::BatchFault* batch_fault = nullptr;  // the batch's kernel error flag, instead of the solver's
    uint64_t faults_seen = 0;       // of batch_fault->count
};

namespace lbm_detail {

int fail(int status, const char* fmt, ...);
int cuda_fail(cudaError_t e, const char* what);
int elem_bytes(int storage);
int value_bytes(int storage);
// Default register variant of a domain.
int default_variant(int storage, const lbm::Grid& g);
// Default register variant of the batch kernel for domains of that many interior
// cells together.
int default_batch_variant(int storage, long long cells);
// Creates a solver; with `external_dd` its populations live there (a batch
// pool) and are initialised but never freed by the solver.
// x1_align, pitch_align: 32, 0 (the default layout) or those of batch pools'
// packed rows (see make_grid).
int create_solver(const lbm_params* prm, void* external_dd, lbm_solver** out, int x1_align = 32, int pitch_align = 0);
void destroy_solver(lbm_solver* s);
int* err_flag(lbm_solver* s);
// Two device words of the solver: [0] the first step of a graph replay,
// [1] always zero (the base of directly launched steps).
uint32_t* step_words(lbm_solver* s);
int check_kernel_flag(lbm_solver* s);

// Runs an entry point's body with C++ exceptions turned into status codes,
// since none may cross the C interface: a host buffer too large for memory
// (a checkpoint or VTK file of a big domain) throws std::bad_alloc.
template <class Body>
int guarded(const char* entry, Body&& body)
{
    try {
        return body();
    } catch (const std::bad_alloc&) {
        return fail(LBM_ERR_OUT_OF_MEMORY, "%s: host allocation failed", entry);
    } catch (const std::exception& e) {
        return fail(LBM_ERR_IO, "%s: %s", entry, e.what());
    }
}

// Largest domain any entry point accepts, halo included: 2^40 cells, far
// beyond device memory (8 bytes x 19 slots x 2^40 cells is 167 TB) and small
// enough that no element or byte count derived from it overflows 64 bits.
constexpr long long kMaxDomainCells = 1LL << 40;
// Each axis in [1, 2^20] and (nx+2)(ny+2)(nz+2) <= kMaxDomainCells.
inline bool domain_size_ok(const int32_t size[3])
{
    long long cells = 1;
    for (int d = 0; d < 3; ++d) {
        if (size[d] <= 0 || size[d] > (1 << 20)) return false;
        cells *= (long long)size[d] + 2;  // < 2^40 * (2^20 + 3) < 2^63
        if (cells > kMaxDomainCells) return false;
    }
    return true;
}

}  // namespace lbm_detail
