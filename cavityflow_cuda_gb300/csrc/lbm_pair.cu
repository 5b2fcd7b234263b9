// lbm_pair.cu -- launches of the two-steps-in-one-pass kernels (lbm_pair.cuh).
#include <cuda.h>
#include <cudaTypedefs.h>

#include "lbm_kernels.h"
#include "lbm_pair.cuh"

namespace lbm {

namespace {

// Tiles of 64 cells (a warp's pairs are one row) by 8 rows for FP32 (20 warps
// at 96 registers) and by 10 for the 16-bit storages (24 warps at 80: more
// warps and fewer frame rows; F16SR 87.4 GLUP/s at 384^3 against 83.6 with 8
// rows, where FP32 spills and falls from 76 to 68).  32 x 8 and 32 x 4 tiles in
// one to three blocks a SM collide more frame cells and ran 15-30 % slower.
// Stages: as many as shared memory holds, up to five.
constexpr int kTX = 64;
template <class St>
struct Shape {
    static constexpr int TY = sizeof(typename St::bits) == 4 ? 8 : 10;
    static constexpr int NST = sizeof(typename St::bits) == 4 ? 4 : 5;
};
int tile_rows(int elem) { return elem == 4 ? Shape<F32>::TY : Shape<F16S>::TY; }

PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            p = nullptr;
        }
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }();
    return fn;
}

int sm_count()
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return sms;
}

// Tiles, and the planes of a z chunk.  A block's time goes with the planes it
// brings through its stages: its items times (chunk + 2).  Long chunks repeat
// fewer planes but let neighbouring blocks drift apart until they no longer
// find each other's frames in L2: at 384^3 FP32 chunks of 16 / 32 / 64 planes
// take 1.485 / 1.500 / 1.635 ms a pair, so a chunk's cost grows by 0.5 % a
// plane and 32 is the longest.
struct Split {
    long long tiles_x, tiles, items;
    int zc;
    long long planes;  // of the busiest block
};
Split split(const Grid& g, int elem, int sms)
{
    const int rows = tile_rows(elem);
    Split s;
    s.tiles_x = (g.nx + kTX - 1) / kTX;
    s.tiles = s.tiles_x * ((g.ny + rows - 1) / rows);
    double best = 0;
    for (int zc = 32; zc >= 8; --zc) {
        const long long chunks = (g.nz + zc - 1) / zc;
        const long long planes = (s.tiles * chunks + sms - 1) / sms * (zc + 2);
        const double cost = (double)planes * (1.0 + 0.005 * zc);
        if (zc == 32 || cost < best) {
            best = cost;
            s.zc = zc;
            s.items = s.tiles * chunks;
            s.planes = planes;
        }
    }
    return s;
}

template <class St>
cudaError_t launch(const void* in, void* out, const Grid& g, const Params& p, int lid_y, int* work, int* err,
                   cudaStream_t st)
{
    using bits = typename St::bits;
    constexpr int TY = Shape<St>::TY, NST = Shape<St>::NST;
    using S = PairShape<St, kTX, TY, NST>;
    const auto encode = encode_fn();
    const int sms = sm_count();
    if (!encode || sms < 1) return cudaErrorNotSupported;
    constexpr cuuint64_t eb = sizeof(bits);
    const cuuint64_t dims[4] = {(cuuint64_t)g.P, (cuuint64_t)g.ny + 2, (cuuint64_t)g.nz + 2, (cuuint64_t)Q};
    const cuuint64_t strides[3] = {(cuuint64_t)g.P * eb, (cuuint64_t)g.PY * eb, (cuuint64_t)g.S * eb};
    const cuuint32_t box[4] = {(cuuint32_t)S::W, TY + 2, 1, (cuuint32_t)Q}, unit[4] = {1, 1, 1, 1};
    CUtensorMap map;
    if (encode(&map, eb == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 4,
               const_cast<void*>(in), dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return cudaErrorInvalidValue;
    auto kern = pair_step<St, kTX, TY, NST>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
    if (e != cudaSuccess) return e;
    const Split s = split(g, (int)eb, sms);
    const PairWork w{(int)s.tiles_x, (int)s.tiles, (int)s.items, s.zc, work};
    const int grid = s.items < sms ? (int)s.items : sms;
    return launch_step(kern, dim3((unsigned)grid), S::THREADS, st, S::SMEM, map, pair_slots(out, g, (int)eb), g,
                       (float)p.inv_tau, (float)p.lid_u, lid_y, p.wall_y, p.step_base, p.step_off, w, err);
}

}  // namespace

bool pair_step_pays(int storage, const Grid& g)
{
    if (storage < 1 || storage > 4) return false;
    const int eb = storage_elem_bytes(storage);
    // the copies' 16-byte alignment, 32-bit offsets into a slot, 32-bit item numbers
    if (!default_layout(g, eb) || (unsigned long long)g.S * eb >= (1ull << 32) || !encode_fn()) return false;
    const int sms = sm_count();
    if (sms < 1) return false;
    const Split s = split(g, eb, sms);
    if (s.items > (1ll << 30)) return false;
    // Measured on GB300, microseconds: a plane of a block, and the separate
    // kernels' cells per microsecond from memory and, while the state fits L2,
    // from there (the pair kernel works on two arrays and so never does).
    static const double plane[5] = {0, 1.80, 1.70, 1.67, 1.96};
    static const double rate[5] = {0, 43000, 80000, 80000, 79000};
    static const double rate_l2[5] = {0, 54000, 75000, 75000, 70000};
    const double state = (double)Q * (double)g.S * eb;
    const double cells = (double)g.nx * g.ny * g.nz;
    const double separate = 2.0 * cells / (state < 100e6 ? rate_l2 : rate)[storage];
    return 6.0 + (double)s.planes * plane[storage] < 0.97 * separate;
}

cudaError_t launch_pair_step(int storage, const void* in, void* out, const Grid& g, const Params& p, int lid_y,
                             int* work, int* err, cudaStream_t st)
{
    add_launches(1);
    switch (storage) {
    case 1: return launch<F32>(in, out, g, p, lid_y, work, err, st);
    case 2: return launch<F16S>(in, out, g, p, lid_y, work, err, st);
    case 3: return launch<BF16S>(in, out, g, p, lid_y, work, err, st);
    case 4: return launch<F16SR>(in, out, g, p, lid_y, work, err, st);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace lbm
