// lbm_pair.cu -- launches of the two-steps-in-one-pass kernels (lbm_pair.cuh).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstring>
#include <functional>
#include <queue>
#include <vector>

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

// The map of a domain's populations for boxes of `slots` slots, `rows` rows of
// `row` elements.
template <class St>
bool make_map(CUtensorMap& map, const void* in, const Grid& g, int row, int rows, int slots)
{
    const auto encode = encode_fn();
    if (!encode) return false;
    constexpr cuuint64_t eb = sizeof(typename St::bits);
    const cuuint64_t dims[4] = {(cuuint64_t)g.P, (cuuint64_t)g.ny + 2, (cuuint64_t)g.nz + 2, (cuuint64_t)Q};
    const cuuint64_t strides[3] = {(cuuint64_t)g.P * eb, (cuuint64_t)g.PY * eb, (cuuint64_t)g.S * eb};
    const cuuint32_t box[4] = {(cuuint32_t)row, (cuuint32_t)rows, 1, (cuuint32_t)slots}, unit[4] = {1, 1, 1, 1};
    return encode(&map, eb == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 4,
                  const_cast<void*>(in), dims, strides, box, unit, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <class St, bool BATCH>
cudaError_t launch(const CUtensorMap& map, const PairCtx& one, const PairWork& w, const uint32_t* step_base,
                   uint32_t step_off, int sms, int* err, cudaStream_t st)
{
    constexpr int TY = Shape<St>::TY, NST = Shape<St>::NST;
    using S = PairShape<St, kTX, TY, NST, BATCH>;
    auto kern = pair_step<St, kTX, TY, NST, BATCH>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return e;
    }
    const int grid = w.items < sms ? w.items : sms;
    return launch_step(kern, dim3((unsigned)grid), S::THREADS, st, S::SMEM, map, one, step_base, step_off, w, err);
}

template <class St>
cudaError_t launch_one(const void* in, void* out, const Grid& g, const Params& p, int lid_y, int* work, int* err,
                       cudaStream_t st, uint64_t limit_ns)
{
    constexpr int TY = Shape<St>::TY, eb = (int)sizeof(typename St::bits);
    const int sms = sm_count();
    CUtensorMap map;
    if (sms < 1 || !make_map<St>(map, in, g, pair_row<St>(kTX), TY + 2, Q)) return cudaErrorNotSupported;
    const Split s = split(g, eb, sms);
    const PairCtx one{g, pair_slots(out, g, eb), {kTX, TY, pair_row<St>(kTX)}, (int)s.tiles_x, (int)s.tiles, s.zc, 0,
                      (float)p.inv_tau, (float)p.lid_u, lid_y, p.wall_y};
    const PairWork w{(int)s.items, limit_ns, work, nullptr, nullptr, nullptr, nullptr};
    return launch<St, false>(map, one, w, p.step_base, p.step_off, sms, err, st);
}

// Tiles for a domain of a batch (FP32): the shape whose planes of the whole
// domain take the least time.  A plane's time, fitted to 45 shapes from 12 x 32
// to 128 x 3 (7 % off on average): its cells', and its rows', which a warp's
// accesses straddle and the copies bring one by one.  Microseconds, GB300, whole
// chip busy, boxes of one tile a row, all of whose tiles have both x walls: 64 x 8
// 2.5-2.8 (2.1 in a large box), 96 x 5 2.65, 48 x 10 2.5-2.7, 32 x 16 3.1-3.4, 14 x
// 32 3.8.
template <class St>
PairDims batch_dims(const Grid& g, double& plane)
{
    constexpr int TY = Shape<St>::TY, NST = Shape<St>::NST;
    PairDims best{0, 0, 0};
    double best_cost = 0;
    for (int nt = 1, last = 0; nt <= g.nx; ++nt) {
        const int tx = ((g.nx + nt - 1) / nt + 1) / 2 * 2;
        if (tx < 8 && nt > 1) break;
        if (tx == last || tx > (nt == 1 ? 96 : kTX)) continue;  // wider ones leave room for few rows
        last = tx;
        int ty = 0;
        while (pair_dims_fit<St, kTX, TY, NST>(tx, ty + 1)) ++ty;
        if (ty == 0) continue;
        const int rows = (g.ny + ty - 1) / ty;
        ty = (g.ny + rows - 1) / rows;
        const double cost = std::max(2.3, 0.0046 * tx * ty + 0.0546 * (ty + 2));
        const double total = cost * rows * ((g.nx + tx - 1) / tx);
        if (best.tx == 0 || total < best_cost) {
            best = {tx, ty, pair_row<St>(tx)};
            best_cost = total;
            plane = cost;
        }
    }
    return best;
}

template <class St>
void plan_batch(const BatchDomain* doms, int count, PairBatchPlan& plan)
{
    constexpr int eb = (int)sizeof(typename St::bits);
    const int sms = sm_count();
    if (sms < 1 || !encode_fn()) return;
    std::vector<PairDomain> table((size_t)count);
    std::vector<double> plane((size_t)count);
    double cells = 0, state = 0;
    for (int i = 0; i < count; ++i) {
        const BatchDomain& b = doms[i];
        PairDomain& d = table[(size_t)i];
        if (b.g.P * eb % 16 != 0 || (unsigned long long)b.g.S * eb >= (1ull << 32) || b.step0 != 0) return;
        d.g = b.g;
        d.offset = b.offset;
        d.dims = batch_dims<St>(b.g, plane[(size_t)i]);
        if (d.dims.tx == 0) return;
        d.tiles_x = (b.g.nx + d.dims.tx - 1) / d.dims.tx;
        d.tiles = d.tiles_x * ((b.g.ny + d.dims.ty - 1) / d.dims.ty);
        d.inv_tau = (float)b.inv_tau;
        d.lid_u = (float)b.lid_u;
        d.lid_y = b.lid_y;
        d.wall_y = b.wall_y;
        cells += (double)b.g.nx * b.g.ny * b.g.nz;
        state += (double)Q * (double)b.g.S * eb;
    }
    // Chunks: long ones repeat fewer planes, short ones fill the chip and its last
    // turns.  The longest items come first, so that the last ones to run are short.
    auto chunk = [&](const PairDomain& d, int zmax) {
        const int n = (d.g.nz + zmax - 1) / zmax;
        return (d.g.nz + n - 1) / n;
    };
    auto count_of = [&](const PairDomain& d, int zc) { return (long long)d.tiles * ((d.g.nz + zc - 1) / zc); };
    std::vector<int> order((size_t)count), best_order;
    std::vector<double> cost((size_t)count);
    double best = 0;
    int best_z = 0;
    for (const int zmax : {32, 24, 16, 12, 8}) {
        long long items = 0;
        double total = 0;
        for (int i = 0; i < count; ++i) {
            const PairDomain& d = table[(size_t)i];
            const int zc = chunk(d, zmax);
            order[(size_t)i] = i;
            cost[(size_t)i] = plane[(size_t)i] * (zc + 2) + 2.0;
            items += count_of(d, zc);
            total += (double)count_of(d, zc) * cost[(size_t)i];
        }
        if (items > (1 << 24)) return;
        std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return cost[(size_t)a] > cost[(size_t)b]; });
        double time = total / sms;
        if (items <= 64 * sms) {  // otherwise the last turn does not matter
            std::priority_queue<double, std::vector<double>, std::greater<double>> free_at;
            for (int i = 0; i < sms; ++i) free_at.push(0);
            time = 0;
            for (const int i : order)
                for (long long n = count_of(table[(size_t)i], chunk(table[(size_t)i], zmax)); n > 0; --n) {
                    const double end = free_at.top() + cost[(size_t)i];
                    free_at.pop();
                    free_at.push(end);
                    time = std::max(time, end);
                }
        }
        if (best_z == 0 || time < best) {
            best = time;
            best_z = zmax;
            best_order = order;
        }
    }
    // Measured: 0.86-1.0 of `best` for 26 batches from 8 cavities of 8 .. 96 cells an edge to 610 of 32^3, where the
    // batch kernels step 34-38 cells a nanosecond from memory and 45 from L2.
    if (4.0 + 0.95 * best >= 0.98 * 2.0 * cells / (state < 100e6 ? 45000 : 36000)) return;
    int items = 0;
    std::vector<int> domain_of;
    for (const int i : best_order) {
        PairDomain& d = table[(size_t)i];
        d.zc = chunk(d, best_z);
        d.item0 = items;
        const int n = (int)count_of(d, d.zc);
        items += n;
        domain_of.insert(domain_of.end(), (size_t)n, i);
    }
    plan.maps[0] = 0;
    plan.maps[1] = (size_t)count * sizeof(CUtensorMap);
    plan.domains = 2 * plan.maps[1];
    plan.domain_of = plan.domains + table.size() * sizeof(PairDomain);
    plan.image.resize(plan.domain_of + domain_of.size() * sizeof(int));
    std::memcpy(plan.image.data() + plan.domains, table.data(), table.size() * sizeof(PairDomain));
    std::memcpy(plan.image.data() + plan.domain_of, domain_of.data(), domain_of.size() * sizeof(int));
    plan.items = items;
}

template <class St>
bool bind_batch(const void* pool, const void* pool2, PairBatchPlan& plan)
{
    const size_t count = plan.maps[1] / sizeof(CUtensorMap);
    for (size_t i = 0; i < count; ++i) {
        PairDomain d;
        std::memcpy(&d, plan.image.data() + plan.domains + i * sizeof(d), sizeof(d));
        for (int k = 0; k < 2; ++k) {
            CUtensorMap map;
            const char* base = static_cast<const char*>(k ? pool2 : pool) + d.offset * (long long)sizeof(typename St::bits);
            if (!make_map<St>(map, base, d.g, d.dims.w, d.dims.ty + 2, 1)) return false;
            std::memcpy(plan.image.data() + plan.maps[k] + i * sizeof(map), &map, sizeof(map));
        }
    }
    return true;
}

template <class St>
cudaError_t launch_batch(const PairBatchPlan& plan, const void* image, bool back, void* out, const uint32_t* step_base,
                         uint32_t step_off, int* work, int* err, cudaStream_t st)
{
    const int sms = sm_count();
    if (sms < 1) return cudaErrorNotSupported;
    const char* const at = static_cast<const char*>(image);
    const PairWork w{plan.items, tma::kWaitLimitNs, work, reinterpret_cast<const PairDomain*>(at + plan.domains),
                     reinterpret_cast<const int*>(at + plan.domain_of),
                     reinterpret_cast<const CUtensorMap*>(at + plan.maps[back ? 1 : 0]), out};
    const CUtensorMap no_map{};
    const PairCtx no_domain{};
    return launch<St, true>(no_map, no_domain, w, step_base, step_off, sms, err, st);
}

}  // namespace

void plan_pair_batch(int storage, const BatchDomain* doms, int count, PairBatchPlan& plan)
{
    plan = PairBatchPlan{};
    if (storage == 1) plan_batch<F32>(doms, count, plan);
}

bool bind_pair_batch(int storage, const void* pool, const void* pool2, PairBatchPlan& plan)
{
    return storage == 1 && bind_batch<F32>(pool, pool2, plan);
}

cudaError_t launch_pair_batch(int storage, const PairBatchPlan& plan, const void* image, bool back, void* out,
                              const uint32_t* step_base, uint32_t step_off, int* work, int* err, cudaStream_t st)
{
    if (storage != 1) return cudaErrorInvalidValue;
    add_launches(1);
    return launch_batch<F32>(plan, image, back, out, step_base, step_off, work, err, st);
}

bool pair_step_runs(int storage, const Grid& g)
{
    if (storage < 1 || storage > 4) return false;
    const int eb = storage_elem_bytes(storage);
    // the copies' 16-byte alignment, 32-bit offsets into a slot, 32-bit item numbers
    if (!default_layout(g, eb) || (unsigned long long)g.S * eb >= (1ull << 32) || !encode_fn()) return false;
    const int sms = sm_count();
    return sms >= 1 && split(g, eb, sms).items <= (1ll << 30);
}

bool pair_step_pays(int storage, const Grid& g)
{
    if (!pair_step_runs(storage, g)) return false;
    const int eb = storage_elem_bytes(storage), sms = sm_count();
    // Microseconds of a pair, fitted to 2350 boxes of 0.3 to 30 million cells with axes up to 8 times off the cube's, GB300.
    //
    // Separate kernels (2 % off, one standard deviation): cells at a rate from memory and at one from L2, in proportion
    // while the state is between two sizes; from memory a row costs `row` cells more, and so does what its last vector
    // leaves unused, everywhere.
    //
    // This kernel (4 % off): the busiest block's planes, of which those beyond an even share count less, since blocks
    // take items as they get done, and a fifth of an item for the last one's start, two fifths for 16-bit rows of an odd
    // number of cells, whose ends take longer than other tiles; more for tiles with an x wall (the copying warp brings
    // the wall slots), for the row ends of odd rows, and for rows that do not fill their tile.
    //
    // What is asked of the ratio is what no box of that set got slower with by more than 1 %; for rows of whole tiles,
    // where the model is better, of another 600.
    // F16SR 291 x 129 x 161: 180 us by pairs, 170 without; F32 37 x 157 x 177: 63 and 57; F16SR 128^3 58.2 and 59.7.
    struct Model {
        double plane, wall, odd, most;                    // this kernel
        double start, l2, memory, row, unused, from, to;  // the others
    };
    static const Model models[5] = {{},
                                    {1.80, 0.22, 0.10, 1.08, 2.9, 63100, 43800, 7.6, 0.83, 80e6, 120e6},
                                    {1.60, 0.13, 0.20, 0.96, 5.6, 100200, 84100, 16.3, 1.29, 70e6, 130e6},
                                    {1.58, 0.13, 0.15, 0.97, 6.8, 110400, 85600, 17.5, 1.21, 60e6, 130e6},
                                    {1.81, 0.12, 0.25, 0.95, 8.6, 103800, 81700, 14.1, 1.17, 70e6, 120e6}};
    const Model& m = models[storage];
    const Split s = split(g, eb, sms);
    const double cells = (double)g.nx * g.ny * g.nz, state = (double)Q * (double)g.S * eb;
    const int vec = 16 / eb;
    const double unused = (double)((g.nx + vec - 1) / vec * vec) / g.nx - 1.0;
    const double memory = std::min(1.0, std::max(0.0, (state - m.from) / (m.to - m.from)));
    const double separate = m.start + 2.0 * cells * ((1.0 - memory) / m.l2 +
                                                     (memory * (1.0 + m.row / g.nx) + m.unused * unused) / m.memory);
    const double chunks = (double)((g.nz + s.zc - 1) / s.zc);
    const double even = (double)s.tiles * (g.nz + 2.0 * chunks) / sms;
    double more = 1.0 + m.wall * std::min(1.0, 2.0 / (double)s.tiles_x);
    if (g.nx % 2) more += m.odd / (double)s.tiles_x + (storage == 4 ? 0.06 : 0.0);
    if (g.nx < kTX) more *= eb == 2 ? 1.25 : 1.15;  // 16 bits, 58 .. 62 wide: up to 1.2 times what the rest says
    const double start = g.nx % 2 && eb == 2 ? 0.4 : 0.2;
    const double pairs = 1.4 + m.plane * ((0.95 * even + 0.75 * ((double)s.planes - even)) * more + start * (s.zc + 2));
    return pairs < (g.nx % kTX == 0 ? std::max(1.0, m.most) : m.most) * separate;
}

cudaError_t launch_pair_step(int storage, const void* in, void* out, const Grid& g, const Params& p, int lid_y,
                             int* work, int* err, cudaStream_t st, int64_t wait_limit_ns)
{
    add_launches(1);
    const uint64_t limit = wait_limit_ns < 0 ? tma::kWaitLimitNs : (uint64_t)wait_limit_ns;
    switch (storage) {
    case 1: return launch_one<F32>(in, out, g, p, lid_y, work, err, st, limit);
    case 2: return launch_one<F16S>(in, out, g, p, lid_y, work, err, st, limit);
    case 3: return launch_one<BF16S>(in, out, g, p, lid_y, work, err, st, limit);
    case 4: return launch_one<F16SR>(in, out, g, p, lid_y, work, err, st, limit);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace lbm
