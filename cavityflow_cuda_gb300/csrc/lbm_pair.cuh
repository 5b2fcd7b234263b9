// lbm_pair.cuh -- two time steps (alpha, then beta) of the box cavity in one
// pass over the populations.
//
// alpha_fast and beta_fast_* each read and write every population once, and
// stream at 0.97 of the copy bandwidth: a pair costs two passes.  pair_step
// reads the state once from `in` and writes the state two steps later to
// `out`, another array of the same layout, so a pair costs one pass (two
// pairs bring the state back to the first array).
//
// A block owns a tile of TX x TY cells and marches along z.  Per plane:
//   1. a warp has TMA bring the 19 slots of the tile and of a one-cell frame
//      around it into a shared-memory stage (one box a plane; for batches a box a slot);
//   2. the alpha threads collide tile and frame in place: population k of a
//      cell goes to slot opp(k) of that cell, wall cells stay as they are,
//      exactly as alpha leaves the array (the frame's cells are collided again
//      by the neighbouring blocks: the price of not waiting for them);
//   3. the beta threads pull what beta pulls from this plane: the five slots
//      with c_z = +1 belong to their cells one plane below, the nine with
//      c_z = 0 to their cells of this plane, the five with c_z = -1 to their
//      cells one plane above.  They wait in registers until a cell has all 19;
//      then it collides and pushes population k to slot k at x + c_k of `out`.
// Slot k of a cell whose neighbour x - c_k is a wall is written by alpha alone
// (nobody pushes into it): the copying warp takes it from the stage to `out`
// when beta is done with the plane.  So `out` gets every slot that a later step reads; slots that no step reads keep
// what they held.  Results are bit-identical to the separate kernels.
//
// The three kinds of threads work on different planes at the same time, a ring
// of stages between them: with all threads first in alpha and then in beta, a
// block's memory and arithmetic phases took turns and a pair was no faster
// than two separate steps (2.61 ms at 384^3 FP32 against 2.58).  A thread owns
// two cells and collides them with paired FP32 instructions (add/mul/fma.
// rn.f32x2: the same IEEE operation on both cells, half the instructions).
//
// Measured on GB300 at 384^3 (ms a pair, separate kernels -> this one): FP32
// 2.58 -> 1.49 (76.0 GLUP/s; 93 % of the copy bandwidth for the bytes it moves,
// 1.11x its array in and 1.0x out), F16S 1.39 -> 1.07 and BF16S 1.38 -> 1.055 (107
// GLUP/s), F16SR 1.41 -> 1.18 (95.7 GLUP/s; its dither is a fifth of its
// instructions).  The 16-bit storages are bound by their instructions (55-62 %
// of the issue slots used, with 24 warps a SM), not by memory.
//
// Batches (FP32): the items of all domains in one launch, the longest first, with
// the tiles of each domain as they fit it best (batch_dims in lbm_pair.cu) and a
// domain's layout and parameters in shared memory.  Same kernel, BATCH: with the
// whole chip busy (384^3, a batch of one) a full tile's plane takes 2.1 us instead
// of 1.9, 0.1 of it for 19 copies in place of one and for addresses from shared
// memory, the rest for rows that start 8 bytes past a sector.  GLUP/s, the separate
// kernels -> this one: 512 cavities of 16 .. 96 cells an edge 34.3 -> 50.4, 76 of
// 64^3 37 -> 54, 610 of 32^3 34.7 -> 45.  The 16-bit storages stay with the separate kernels:
// they move half the bytes and ran at 0.75 .. 1.0 of their speed here.
#pragma once

#include <cstdint>
#include <type_traits>
#include <cuda.h>

#include "lbm_core.cuh"
#include "lbm_fast.cuh"
#include "lbm_kernels.h"
#include "lbm_tma.cuh"

namespace lbm {

// ---------------------------------------------------------------------------
// Two FP32 values in one 64-bit register pair.
// ---------------------------------------------------------------------------
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2_make(float lo, float hi)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ F2 f2_both(float a) { return f2_make(a, a); }
__device__ __forceinline__ void f2_split(F2 a, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b)
{
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

// Product with a constant, as two scalar multiplies: given a constant operand,
// ptxas contracts mul.rn.f32x2 and the add or sub that follows into one fused
// multiply-add, which changes the result; the scalar mul.rn.f32 it leaves alone.
// The FP32 pipe takes as long for two scalar operations as for a paired one.
// Paired products of two variables come out unfused so far, but nothing says that
// they must where a paired sum follows, so such a sum is scalar (f2_sum3: 0.2 % of
// the FP32 kernel's time; scalar products 0.8 %; fused multiply-adds with -0 in
// place of the products do not do, ptxas makes products of them and contracts
// those).
__device__ __forceinline__ F2 f2_scale(float c, F2 a)
{
    float lo, hi;
    f2_split(a, lo, hi);
    return f2_make(__fmul_rn(c, lo), __fmul_rn(c, hi));
}

__device__ __forceinline__ F2 f2_sum3(F2 a, F2 b, F2 c)
{
    float a0, a1, b0, b1, c0, c1;
    f2_split(a, a0, a1);
    f2_split(b, b0, b1);
    f2_split(c, c0, c1);
    return f2_make(__fadd_rn(__fadd_rn(a0, b0), c0), __fadd_rn(__fadd_rn(a1, b1), c1));
}

// relax_pair (lbm_core.cuh) on two cells: the same operations in the same
// order, except that P + (-3 s) is written P - 3 s, which is the same value.
__device__ __forceinline__ void relax_pair2(F2& fp, F2& fm, float w, F2 P, F2 s, float inv_tau)
{
    const F2 s2 = s * s;
    const F2 t = f2_scale(4.5f, s2);
    const F2 a = f2_scale(3.0f, s);
    const F2 ep = f2_scale(w, (P + a) + t);
    const F2 em = f2_scale(w, (P - a) + t);
    fp = fp + f2_scale(inv_tau, ep - fp);
    fm = fm + f2_scale(inv_tau, em - fm);
}

// collide_fluid<float> on two cells.
__device__ __forceinline__ void collide_fluid2(F2* f, float inv_tau)
{
    F2 r = f[0], x = f[0], y, z;
    r = r + f[1];  x = x - f[1];
    r = r + f[2];  y = f[2];
    r = r + f[3];  y = y - f[3];
    r = r + f[4];  x = x + f[4];  y = y + f[4];
    r = r + f[5];  x = x - f[5];  y = y - f[5];
    r = r + f[6];  x = x + f[6];  y = y - f[6];
    r = r + f[7];  x = x - f[7];  y = y + f[7];
    r = r + f[8];  x = x + f[8];  z = f[8];
    r = r + f[9];  x = x - f[9];  z = z - f[9];
    r = r + f[10]; x = x + f[10]; z = z - f[10];
    r = r + f[11]; x = x - f[11]; z = z + f[11];
    r = r + f[12]; y = y + f[12]; z = z + f[12];
    r = r + f[13]; y = y - f[13]; z = z - f[13];
    r = r + f[14]; y = y + f[14]; z = z - f[14];
    r = r + f[15]; y = y - f[15]; z = z + f[15];
    r = r + f[16]; z = z + f[16];
    r = r + f[17]; z = z - f[17];
    r = r + f[18];
    const F2 P = r - f2_scale(1.5f, f2_sum3(x * x, y * y, z * z));
    constexpr float wa = 1.0f / 18.0f, wd = 1.0f / 36.0f;
    relax_pair2(f[0], f[1], wa, P, x, inv_tau);
    relax_pair2(f[2], f[3], wa, P, y, inv_tau);
    relax_pair2(f[4], f[5], wd, P, x + y, inv_tau);
    relax_pair2(f[6], f[7], wd, P, x - y, inv_tau);
    relax_pair2(f[8], f[9], wd, P, x + z, inv_tau);
    relax_pair2(f[10], f[11], wd, P, x - z, inv_tau);
    relax_pair2(f[12], f[13], wd, P, y + z, inv_tau);
    relax_pair2(f[14], f[15], wd, P, y - z, inv_tau);
    relax_pair2(f[16], f[17], wa, P, z, inv_tau);
    f[18] = f[18] + f2_scale(inv_tau, f2_scale(1.0f / 3.0f, P) - f[18]);
}

// relax_pair_shifted / collide_shifted on two cells.
__device__ __forceinline__ void relax_pair_shifted2(F2& sp, F2& sm, float w3, float w45, F2 wP, F2 u, F2 omega)
{
    const F2 even = f2_fma(f2_both(w45), u * u, wP);
    const F2 odd = f2_scale(w3, u);
    sp = f2_fma(omega, (even + odd) - sp, sp);
    sm = f2_fma(omega, (even - odd) - sm, sm);
}

template <int E>
__device__ __forceinline__ void collide_shifted2(F2* s, F2 omega)
{
    const F2 a01 = s[0] + s[1], d01 = s[0] - s[1];
    const F2 a23 = s[2] + s[3], d23 = s[2] - s[3];
    const F2 a45 = s[4] + s[5], d45 = s[4] - s[5];
    const F2 a67 = s[6] + s[7], d67 = s[6] - s[7];
    const F2 a89 = s[8] + s[9], d89 = s[8] - s[9];
    const F2 a1011 = s[10] + s[11], d1011 = s[10] - s[11];
    const F2 a1213 = s[12] + s[13], d1213 = s[12] - s[13];
    const F2 a1415 = s[14] + s[15], d1415 = s[14] - s[15];
    const F2 a1617 = s[16] + s[17], d1617 = s[16] - s[17];
    const F2 drho = ((a01 + a23) + (a45 + a67)) + ((a89 + a1011) + (a1213 + a1415)) + (a1617 + s[18]);
    const F2 jx = ((d01 + d45) + (d67 + d89)) + d1011;
    const F2 jy = ((d23 + d45) - d67) + (d1213 + d1415);
    const F2 jz = ((d89 - d1011) + (d1213 - d1415)) + d1617;
    const F2 vel2 = f2_fma(jz, jz, f2_fma(jy, jy, jx * jx));
    constexpr float inv_scale = 1.0f / (float)(1u << E);
    const F2 P = f2_fma(f2_both(-1.5f * inv_scale), vel2, drho);
    constexpr float wa = 1.0f / 18.0f, wd = 1.0f / 36.0f;
    const F2 waP = f2_scale(wa, P), wdP = f2_scale(wd, P);
    constexpr float wa3 = 3.0f * wa, wa45 = (4.5f * wa) * inv_scale, wd3 = 3.0f * wd, wd45 = (4.5f * wd) * inv_scale;
    relax_pair_shifted2(s[0], s[1], wa3, wa45, waP, jx, omega);
    relax_pair_shifted2(s[2], s[3], wa3, wa45, waP, jy, omega);
    relax_pair_shifted2(s[4], s[5], wd3, wd45, wdP, jx + jy, omega);
    relax_pair_shifted2(s[6], s[7], wd3, wd45, wdP, jx - jy, omega);
    relax_pair_shifted2(s[8], s[9], wd3, wd45, wdP, jx + jz, omega);
    relax_pair_shifted2(s[10], s[11], wd3, wd45, wdP, jx - jz, omega);
    relax_pair_shifted2(s[12], s[13], wd3, wd45, wdP, jy + jz, omega);
    relax_pair_shifted2(s[14], s[15], wd3, wd45, wdP, jy - jz, omega);
    relax_pair_shifted2(s[16], s[17], wa3, wa45, waP, jz, omega);
    s[18] = f2_fma(omega, f2_scale(1.0f / 3.0f, P) - s[18], s[18]);
}

// One step's cell rule on two cells of a row: wall correction, then the lid's
// equilibrium or the collision.
template <class St>
__device__ __forceinline__ void cell_rule2(F2* f, bool lid, bool wall, float inv_tau, float lid_u)
{
    if (wall) {
        const F2 du = f2_both(wall_shift<St>(lid_u));
        f[5] = f[5] - du;
        f[6] = f[6] + du;
    }
    if (lid) {
        float e[Q];
        inject_step<St>(e, St::shifted ? 0.0f : 1.0f, lid_u);
#pragma unroll
        for (int k = 0; k < Q; ++k) f[k] = f2_both(e[k]);
    } else if constexpr (St::shifted) {
        collide_shifted2<St::kStepLog2>(f, f2_both(inv_tau));
    } else {
        collide_fluid2(f, inv_tau);
    }
}

// ---------------------------------------------------------------------------
// Two neighbouring stored populations of a slot: 8 bytes (FP32) or one word.
// ---------------------------------------------------------------------------
template <class St, bool kWide = sizeof(typename St::bits) == 4>
struct Two;

template <class St>
struct Two<St, true> {
    using raw = unsigned long long;
    __device__ static raw load(const float* p) { return *reinterpret_cast<const raw*>(p); }
    __device__ static void store(float* p, raw r) { *reinterpret_cast<raw*>(p) = r; }
    __device__ static raw join(float a, float b) { return f2_make(a, b).v; }
    __device__ static float first(raw r)
    {
        float a, b;
        f2_split(F2{r}, a, b);
        return a;
    }
    __device__ static float second(raw r)
    {
        float a, b;
        f2_split(F2{r}, a, b);
        return b;
    }
    // the cells at p[DX] and p[DX + sep]
    template <int DX>
    __device__ static raw load_at(const float* p, int sep)
    {
        return join(p[DX], p[DX + sep]);
    }
    __device__ static F2 widen(raw r) { return F2{r}; }
    __device__ static raw narrow(F2 v, uint32_t, uint32_t, int) { return v.v; }
};

template <class St>
struct Two<St, false> {
    using raw = uint32_t;
    using bits = unsigned short;
    __device__ static raw load(const bits* p) { return *reinterpret_cast<const raw*>(p); }
    __device__ static void store(bits* p, raw r) { *reinterpret_cast<raw*>(p) = r; }
    __device__ static raw join(bits a, bits b) { return (raw)a | ((raw)b << 16); }
    __device__ static bits first(raw r) { return (bits)(r & 0xffffu); }
    __device__ static bits second(raw r) { return (bits)(r >> 16); }
    // the cells at p[DX] and p[DX + 1], p aligned to a word (sep is 1)
    template <int DX>
    __device__ static raw load_at(const bits* p, int)
    {
        if constexpr (DX == 0) return load(p);
        else if constexpr (DX == 1) return __byte_perm(load(p), load(p + 2), 0x5432);
        else return __byte_perm(load(p - 2), load(p), 0x5432);
    }
    __device__ static F2 widen(raw r) { return f2_make(St::load_step(first(r)), St::load_step(second(r))); }
    __device__ static raw narrow(F2 v, uint32_t h0, uint32_t h1, int k)
    {
        float a, b;
        f2_split(v, a, b);
        return pk_two<St>(pk_pre<St>(a, h0, k), pk_pre<St>(b, h1, k));
    }
};

// Tiles.  A stage holds, of one plane, all 19 slots (SLOT elements apart) of the
// tile's rows and one on either side, from a 16-byte boundary left of the tile's
// left neighbour column to one right of its right neighbour column (TMA copies
// start and end on such boundaries).  The threads are those of TX x TY cells;
// other shapes that need no more of them, and no more room, run on the kernel of
// batches (PairDims), so that the tiles fit each cavity.
template <class St, int TX, int TY, int NST, bool BATCH>
struct PairShape {
    using bits = typename St::bits;
    static_assert(!BATCH || sizeof(bits) == 4, "batches take two steps a pass in FP32 only");
    static constexpr int kAlign = 16 / (int)sizeof(bits);        // elements to a 16-byte boundary
    static constexpr int kUnit = 128 / (int)sizeof(bits);        // of a copy's destination
    static constexpr int kSlot = (TY + 2) * (TX + 2 * kAlign);
    static constexpr int SLOT = BATCH ? (kSlot + kUnit - 1) / kUnit * kUnit : kSlot;
    static constexpr int STAGE = (Q * SLOT + kUnit - 1) / kUnit * kUnit;
    static constexpr int NA = ((TY + 2) * (TX / 2 + 2) + 31) / 32 * 32;  // alpha threads: pairs of tile rows -1 .. TY, the frame's columns
    static constexpr int NB = TY * (TX / 2);                     // beta threads
    static constexpr int THREADS = NA + NB + 32;                 // and the warp that issues the copies
    static constexpr size_t SMEM = (size_t)NST * STAGE * sizeof(bits) + NST * (sizeof(uint64_t) + 2 * sizeof(int));
    static_assert(NB % 32 == 0, "whole warps");
    static_assert(1 + 2 * NST <= 15, "named barriers");
};

// A tile's cells along x (even) and y, and the elements of a stage row.
struct PairDims {
    int tx, ty, w;
};
template <class St>
__host__ __device__ constexpr int pair_row(int tx)
{
    const int align = 16 / (int)sizeof(typename St::bits);
    // the tile's first cell is at most `align` columns in, and one follows its last
    return tx % align == 0 ? tx + 2 * align : (align + tx + 1 + align - 1) / align * align;
}
template <class St, int TX, int TY, int NST>
constexpr bool pair_dims_fit(int tx, int ty)
{
    using S = PairShape<St, TX, TY, NST, true>;
    return tx >= 2 && tx % 2 == 0 && ty >= 1 && (ty + 2) * (tx / 2 + 2) <= S::NA && ty * (tx / 2) <= S::NB &&
           (ty + 2) * pair_row<St>(tx) <= S::SLOT && pair_row<St>(tx) <= 256 && ty + 2 <= 256;
}

// Named barriers, as a producer and a consumer use them: `arrive` does not wait.
__device__ __forceinline__ void named_sync(int id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void named_arrive(int id, int threads)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Where the slots of `out` are: own[k] + o is slot k of the cell at byte o of
// its slot, push[k] + o the place in slot k, one plane below, that the cell
// pushes population k to.  Uniform bases and a 32-bit offset a thread: one
// address per access instead of a 64-bit sum.
struct PairSlots {
    char* own[Q];
    char* push[Q];
};
inline PairSlots pair_slots(void* out, const Grid& g, int elem)
{
    PairSlots s;
    for (int k = 0; k < Q; ++k) {
        s.own[k] = static_cast<char*>(out) + (long long)k * g.S * elem;
        s.push[k] = s.own[k] + ((dir_z(k) - 1) * g.PY + dir_y(k) * g.P + dir_x(k)) * elem;
    }
    return s;
}

// A domain as the threads of the kernel see it.
struct PairCtx {
    Grid g;
    PairSlots slots;
    PairDims dims;       // of its tiles
    int tiles_x, tiles;  // tiles of a row, of a plane
    int zc;              // planes of a chunk
    int item;            // batches: the item in work, counted within the domain
    float inv_tau, lid_u;
    int lid_y, wall_y;
};

// A domain of a batch: PairCtx is made of it when one of its items comes up.
struct PairDomain {
    Grid g;
    long long offset;  // elements from the pool's base
    PairDims dims;
    int tiles_x, tiles, zc;
    int item0;         // its first item
    float inv_tau, lid_u;
    int lid_y, wall_y;
};

// The work of one launch: items, each a tile of a z chunk (of a domain), chunks
// slowest.  Blocks are persistent and take the next item from a counter, so
// that at any time they work on neighbouring tiles of the same planes and find
// each other's frames in L2; a block's copies run ahead into its next item.
struct PairWork {
    int items;
    uint64_t limit_ns;          // of the wait for a copy
    int* next;                  // [0] items taken beyond the first of each block, [1] blocks done; zero between launches
    const PairDomain* domains;  // batches: the domains, the domain of each item, the copies' maps of each
    const int* domain_of;       // domain's array, the array written to
    const CUtensorMap* maps;
    void* out;
};
struct PairItem {
    int x0, y0, za, zb;  // first cell, first and last plane
};
__device__ __forceinline__ PairItem pair_item(const PairCtx& c, const PairDims& d, int item)
{
    const int chunk = item / c.tiles, t = item - chunk * c.tiles;
    const int ty = t / c.tiles_x, tx = t - ty * c.tiles_x;
    const int za = 1 + chunk * c.zc;
    return {1 + tx * d.tx, 1 + ty * d.ty, za, min(c.g.nz, za + c.zc - 1)};
}
// First column of a stage row: the last 16-byte boundary left of the tile's left
// neighbour column.
template <class St>
__device__ __forceinline__ int pair_column(const Grid& g, int x0)
{
    return (g.xoff + x0 - 1) & ~(16 / (int)sizeof(typename St::bits) - 1);
}

// Where the threads find the domain of an item.  One domain: the kernel's
// parameters, tiles of TX x TY.  A batch: shared memory, where the copying warp
// puts it; a block has at most three items between its stages and that warp.
constexpr int kPairContexts = 4;
template <class St, int TX, int TY, bool BATCH>
struct PairSource {
    const PairCtx& one;
    PairCtx* many;
    __device__ __forceinline__ const PairCtx& at(int item) const
    {
        if constexpr (BATCH) return many[item & (kPairContexts - 1)];
        else return one;
    }
    __device__ __forceinline__ PairDims dims(int item) const
    {
        if constexpr (BATCH) return at(item).dims;
        else return {TX, TY, pair_row<St>(TX)};
    }
    __device__ __forceinline__ PairItem item(int n) const
    {
        if constexpr (BATCH) return pair_item(at(n), dims(n), at(n).item);
        else return pair_item(one, dims(n), n);
    }
};

// Waits until the phase with `parity` of `bar` has completed; false when
// limit_ns have passed since its fill was seen to be issued (*issued == parity).
__device__ __forceinline__ bool pair_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns, const volatile int* issued)
{
    constexpr uint32_t kNap = 100000;  // ns the hardware may suspend the thread
    uint64_t deadline = 0;
    for (;;) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(tma::smem_addr(bar)), "r"(parity), "r"(limit_ns < kNap ? (uint32_t)limit_ns : kNap)
            : "memory");
        if (done) return true;
        if (*issued != (int)parity) continue;
        const uint64_t now = tma::now_ns();
        if (deadline == 0) deadline = now + limit_ns;
        if (now >= deadline) return false;
    }
}

// The slots that point away from the low (SIGN 1) or high (-1) wall of an axis.
template <int AXIS, int SIGN>
struct FromFace {
    __host__ __device__ static constexpr bool at(int k) { return (AXIS == 0 ? dir_x(k) : AXIS == 1 ? dir_y(k) : dir_z(k)) == SIGN; }
};

// Index of slot k among the slots of its c_z.
__host__ __device__ constexpr int z_rank(int k)
{
    int n = 0;
    for (int q = 0; q < k; ++q) n += dir_z(q) == dir_z(k);
    return n;
}

// Slots of a tile's plane p that no beta thread writes, as the neighbour they
// would come from is a wall: what alpha left in them goes to `out` as it is.  By
// the copying warp, which has the time, when beta is done with the stage.  Done
// by beta's threads this took the tiles at the walls a fifth longer (ms a pair
// at 384^3, then -> now: BF16S 1.105 -> 1.046, F16SR 1.284 -> 1.208; at 256^3
// 0.343 -> 0.323 and 0.393 -> 0.368), by alpha's even more (1.168, 1.324).
template <class St, int SLOT>
__device__ __forceinline__ void pair_walls(const PairCtx& c, const PairDims& d, const typename St::bits* sb, int x0,
                                           int y0, int p)
{
    using bits = typename St::bits;
    const Grid& g = c.g;
    const int lane = (int)threadIdx.x & 31;
    const int nx = min(d.tx, g.nx + 1 - x0), ny = min(d.ty, g.ny + 1 - y0);
    const bits* const first = sb + d.w + (g.xoff + x0 - pair_column<St>(g, x0));
    const uint32_t off = (uint32_t)(g.idx(x0, y0, p) * (long long)sizeof(bits)), row = (uint32_t)(g.P * (long long)sizeof(bits));
    // columns x .. x + n - 1 of the tile's rows y .. y + m - 1
    auto area = [&](auto face, int x, int n, int y, int m) {
#pragma unroll 1
        for (int i = lane; i < n * m; i += 32) {
            const int yi = y + i / n, xi = x + i % n;
            const bits* const from = first + yi * d.w + xi;
            const uint32_t to = off + (uint32_t)yi * row + (uint32_t)(xi * (int)sizeof(bits));
            static_for<0, Q>([&](auto kc) {
                constexpr int k = decltype(kc)::value;
                if constexpr (decltype(face)::at(k)) *reinterpret_cast<bits*>(c.slots.own[k] + to) = from[k * SLOT];
            });
        }
    };
    if (x0 == 1) area(FromFace<0, 1>{}, 0, 1, 0, ny);
    if (x0 + nx > g.nx) area(FromFace<0, -1>{}, nx - 1, 1, 0, ny);
    if (y0 == 1) area(FromFace<1, 1>{}, 0, nx, 0, 1);
    if (y0 + ny > g.ny) area(FromFace<1, -1>{}, 0, nx, ny - 1, 1);
    if (p == 1) area(FromFace<2, 1>{}, 0, nx, 0, ny);
    if (p == g.nz) area(FromFace<2, -1>{}, 0, nx, 0, ny);
}

// The copying warp: takes items and brings the planes za - 1 .. zb + 1 of each
// into the stages, as beta gives them back.  item_of[s] tells the others which
// item stage s holds (one domain: its number; a batch: the block's how-manieth);
// -1 ends the block.  Fills of stages are counted over the block's life; fill u
// goes into stage u % NST; issued[s] is the parity of u / NST of the last one under
// way or done there.
//
// A block also ends when alpha's wait for a copy runs out: alpha then writes -1
// over the item of that fill, so that all leave at it as at the regular end,
// without another look at the stages or another store to `out`, and this warp
// waits, again bounded, for the copies that are still on their way here.  Alpha's
// clock runs from the issue of the fill: what comes before that, the previous
// kernel's end or beta giving the stage back, is no fault of the copy, and only
// then are all through with the stage's last use, so that nobody reads the -1 for
// another fill or arrives twice on one of its barriers.
template <class St, int TX, int TY, int NST, bool BATCH>
__device__ __forceinline__ void pair_copy(const CUtensorMap* map, const PairSource<St, TX, TY, BATCH>& src,
                                          const PairWork& w, typename St::bits* smem, uint64_t* full, int* item_of,
                                          volatile int* issued)
{
    using S = PairShape<St, TX, TY, NST, BATCH>;
    using bits = typename St::bits;
    const int lane = (int)threadIdx.x & 31;
    const bool lead = lane == 0;
    int stage = 0, item = (int)blockIdx.x, next = 0, seen = -1;
    // lane s: what stage s holds, and whether the tile's plane has walls beside it
    bool walls = false;
    int held_x0 = 0, held_y0 = 0, held_p = 0;
    // the item whose planes are being brought, the plane that comes next
    PairItem it{0, 0, 0, -2};
    PairDims dims{0, 0, 0};
    int n = 0, p = 0, col = 0, fills = 0, last = -1;
    uint32_t phase = 0;
    bool edge = false, all_brought = false;
    // This block takes no more items.  Every block comes here once, the last one leaves the counters as the next launch
    // wants them.
    auto no_more = [&]() {
        all_brought = true;
        if (lead && atomicAdd(&w.next[1], 1) == (int)gridDim.x - 1) {
            w.next[0] = 0;
            w.next[1] = 0;
        }
    };
    // `in`, `out` and the counters are the previous step's until it is complete; the other threads touch global memory
    // only after this warp's first copy has arrived
    wait_previous_step();
    // One turn a fill; after the last, the fill that ends the block, one for each that beta has still to give back.
#pragma unroll 1
    for (int use = 0;; ++use) {
        if (!all_brought && p == it.zb + 2) {  // the next item, while beta is still busy
            if (use > 0) item = __shfl_sync(0xffffffffu, next, 0) + (int)gridDim.x;
            if (item < w.items) {
                n = BATCH ? ++seen : item;
                if constexpr (BATCH) {
                    const int dom = w.domain_of[item];
                    const PairDomain& d = w.domains[dom];
                    PairCtx& c = src.many[n & (kPairContexts - 1)];
                    const Grid g = d.g;
                    static_for<0, Q>([&](auto kc) {
                        constexpr int k = decltype(kc)::value;
                        if (lane == k) {
                            char* const own = static_cast<char*>(w.out) + (d.offset + k * g.S) * (long long)sizeof(bits);
                            c.slots.own[k] = own;
                            c.slots.push[k] =
                                own + ((dir_z(k) - 1) * g.PY + dir_y(k) * g.P + dir_x(k)) * (long long)sizeof(bits);
                        }
                    });
                    if (lane == Q) {
                        c.g = g;
                        c.dims = d.dims;
                        c.tiles_x = d.tiles_x;
                        c.tiles = d.tiles;
                        c.zc = d.zc;
                        c.item = item - d.item0;
                        c.inv_tau = d.inv_tau;
                        c.lid_u = d.lid_u;
                        c.lid_y = d.lid_y;
                        c.wall_y = d.wall_y;
                    }
                    __syncwarp();
                    map = w.maps + dom;
                    if (lead) asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(map) : "memory");
                }
                it = src.item(n);
                dims = src.dims(n);
                const Grid& g = src.at(n).g;
                col = pair_column<St>(g, it.x0);
                edge = it.x0 == 1 || it.y0 == 1 || it.x0 + dims.tx > g.nx || it.y0 + dims.ty > g.ny;
                p = it.za - 1;
            } else {
                no_more();
                last = use;
            }
        }
        if (use >= NST) {
            named_sync(1 + NST + stage, S::NB + 32);  // beta is done with fill use - NST
            const bool at_walls = __shfl_sync(0xffffffffu, (int)walls, stage);
            const int was = *(const volatile int*)&item_of[stage];
            if (was < 0) {  // the block ended there
                if (!all_brought) no_more();
                for (int u = use - NST; u < fills; ++u)  // copies that nobody has waited for
                    pair_wait(&full[u % NST], (uint32_t)(u / NST) & 1u, tma::kWaitLimitNs, &issued[u % NST]);
                return;
            }
            if (at_walls) {
                pair_walls<St, S::SLOT>(src.at(was), src.dims(was), smem + stage * S::STAGE,
                                        __shfl_sync(0xffffffffu, held_x0, stage), __shfl_sync(0xffffffffu, held_y0, stage),
                                        __shfl_sync(0xffffffffu, held_p, stage));
                __syncwarp();
            }
        }
        if (use == last && lead) {
            item_of[stage] = -1;
            tma::mbar_arrive(&full[stage]);
            issued[stage] = (int)phase;
        }
        if (!all_brought) {
            if (lead && p == it.zb) next = atomicAdd(&w.next[0], 1);
            if (lane == stage) {
                held_x0 = it.x0;
                held_y0 = it.y0;
                held_p = p;
                walls = p >= it.za && p <= it.zb && (edge || p == 1 || p == src.at(n).g.nz);
            }
            if (lead) {
                item_of[stage] = n;
                tma::fence_proxy_async();  // alpha's and beta's accesses to the stage, before the copy overwrites it
                tma::mbar_arrive_expect_tx(&full[stage], (uint32_t)(Q * (dims.ty + 2) * dims.w * (int)sizeof(bits)));
                const uint32_t to = tma::smem_addr(smem + stage * S::STAGE), bar = tma::smem_addr(&full[stage]);
                // all slots in one box; a batch's boxes are of many sizes, the slots' places in a stage are not
#pragma unroll 1
                for (int k = 0; k < (BATCH ? Q : 1); ++k)
                    asm volatile(
                        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, "
                        "%4, %5}], [%6];" ::"r"(to + (uint32_t)(k * S::SLOT * (int)sizeof(bits))),
                        "l"(map), "r"(col), "r"(it.y0 - 1), "r"(p), "r"(k), "r"(bar)
                        : "memory");
                issued[stage] = (int)phase;
            }
            ++p;
            ++fills;
        }
        if (++stage == NST) {
            stage = 0;
            phase ^= 1;
        }
    }
}

// Alpha threads: collide the cells of a stage in place.
template <class St, int TX, int TY, int NST, bool BATCH>
__device__ __forceinline__ void pair_alpha(const PairSource<St, TX, TY, BATCH>& src, const uint32_t step,
                                           typename St::bits* __restrict__ smem, uint64_t* full,
                                           int* item_of, const volatile int* issued, const uint64_t limit_ns,
                                           int* __restrict__ err)
{
    using S = PairShape<St, TX, TY, NST, BATCH>;
    using bits = typename St::bits;
    using two = Two<St>;
    const int tid = (int)threadIdx.x;
    bits* own = smem;
    int stage = 0;
    uint32_t phase = 0;
    int item = -2, p = 0, y = 0, xa = 0;  // no item yet
    bool work = false, both = false, lid = false, wall = false;
#pragma unroll 1
    for (;;) {
        // one warp looks for the copy's arrival, the others sleep in a barrier: 11 or 13 warps looking took
        // issue slots from beta's (F16SR 1.276 ms a pair instead of 1.296 at 384^3)
        if (tid < 32 && !pair_wait(&full[stage], phase, limit_ns, &issued[stage])) {
            *(volatile int*)&item_of[stage] = -1;
            atomicOr(err, 4);
        }
        named_sync(1 + 2 * NST, S::NA);
        const int now = *(const volatile int*)&item_of[stage];
        ++p;
        if (now != item) {  // another tile's first plane
            if (now < 0) break;
            item = now;
            const PairItem it = src.item(item);
            const PairDims d = src.dims(item);
            const Grid& g = src.at(item).g;
            // Pairs of tile rows -1 .. ty, then two cells left and two right of each of these rows, of which the frame
            // has the nearer one; the other cell of such a pair is collided from whatever the stage holds, and nothing
            // reads it.
            const int c = tid - (d.ty + 2) * (d.tx / 2);
            const bool column = c >= 0;
            const int ry = column ? (c < d.ty + 2 ? c : c - (d.ty + 2)) : tid / (d.tx / 2);
            const int px = !column ? tid % (d.tx / 2) : c < d.ty + 2 ? -1 : d.tx / 2;
            p = it.za - 1;
            y = it.y0 - 1 + ry;
            xa = it.x0 + 2 * px;
            const int x = column && px < 0 ? xa + 1 : xa;  // the cell that decides
            work = ry <= d.ty + 1 && y >= 1 && y <= g.ny && x >= 1 && x <= g.nx;
            both = column || xa < g.nx;
            lid = y == src.at(item).lid_y;
            wall = y == src.at(item).wall_y;
            own = smem + ry * d.w + (g.xoff + xa - pair_column<St>(g, it.x0));
        }
        const PairCtx& ctx = src.at(item);
        bits* const sb = own + stage * S::STAGE;
        if (p >= 1 && p <= ctx.g.nz && work) {
            uint32_t ha = 0, hb = 0;
            if constexpr (St::stochastic) {
                const uint32_t rh = sr_hash((uint32_t)ctx.g.ref(0, y, p), step);
                ha = sr_cell(rh, xa);
                hb = sr_cell(rh, xa + 1);
            }
            F2 f[Q];
#pragma unroll
            for (int k = 0; k < Q; ++k) f[k] = two::widen(two::load(sb + k * S::SLOT));
            cell_rule2<St>(f, lid, wall, ctx.inv_tau, ctx.lid_u);
            if (both) {
#pragma unroll
                for (int k = 0; k < Q; ++k) two::store(sb + opp(k) * S::SLOT, two::narrow(f[k], ha, hb, k));
            } else {  // the second cell is the wall behind the row's end
#pragma unroll
                for (int k = 0; k < Q; ++k) sb[opp(k) * S::SLOT] = two::first(two::narrow(f[k], ha, hb, k));
            }
        }
        named_arrive(1 + stage, S::NA + S::NB);
        if (++stage == NST) {
            stage = 0;
            phase ^= 1;
        }
    }
    named_arrive(1 + stage, S::NA + S::NB);
}

// Beta threads: pull, collide, push to `out`.
template <class St, int TX, int TY, int NST, bool BATCH>
__device__ __forceinline__ void pair_beta(const PairSource<St, TX, TY, BATCH>& src, const uint32_t step,
                                          typename St::bits* __restrict__ smem, const int* item_of)
{
    using S = PairShape<St, TX, TY, NST, BATCH>;
    using bits = typename St::bits;
    using two = Two<St>;
    using raw = typename two::raw;
    constexpr bool k16 = sizeof(bits) == 2;
    const int tid = (int)threadIdx.x - S::NA;
    const bits* own = smem;
    raw c0[9], m1[5], m2[5];
    int stage = 0, item = -2, p = 0, za = 0, zb = 0, y = 0, xa = 0;  // no item yet
    // The thread's two cells: FP32 half a row apart, so that each access of a warp is runs of 4-byte elements whatever
    // the shift; 16-bit neighbours, one word.
    int SEP = k16 ? 1 : TX / 2, W = pair_row<St>(TX);
    bool tile = false, vb = false, whole_rows = false, lid = false, wall = false;
    uint32_t off = 0, pitch = 0;  // of (xa, y, p) in a slot, of a plane, bytes
#pragma unroll 1
    for (;;) {
        named_sync(1 + stage, S::NA + S::NB);
        const int now = *(const volatile int*)&item_of[stage];
        ++p;
        off += pitch;
        if (now != item) {  // another tile's first plane
            if (now < 0) break;
            item = now;
            const PairItem it = src.item(item);
            const PairDims d = src.dims(item);
            const Grid& g = src.at(item).g;
            const int ry = tid / (d.tx / 2), px = tid % (d.tx / 2);
            if (BATCH) {
                SEP = d.tx / 2;
                W = d.w;
            }
            za = it.za;
            zb = it.zb;
            p = za - 1;
            y = it.y0 + ry;
            xa = it.x0 + (k16 ? 2 * px : px);
            tile = ry < d.ty && y <= g.ny && xa <= g.nx;
            vb = xa + SEP <= g.nx;
            whole_rows = !__any_sync(0xffffffffu, tile && !vb);
            lid = y == src.at(item).lid_y;
            wall = y == src.at(item).wall_y;
            off = (uint32_t)(g.idx(xa, y, p) * (long long)sizeof(bits));
            pitch = (uint32_t)(g.PY * (long long)sizeof(bits));
            own = smem + (ry + 1) * d.w + (g.xoff + xa - pair_column<St>(g, it.x0));
        }
        const PairCtx& ctx = src.at(item);
        const Grid& g = ctx.g;
        const PairSlots& slots = ctx.slots;
        if (tile) {
            const bits* const sb = own + stage * S::STAGE;
            if (p > za) {  // the cells of plane p - 1 have all their populations now
                F2 f[Q];
                static_for<0, Q>([&](auto kc) {
                    constexpr int k = decltype(kc)::value;
                    raw r;
                    if constexpr (dir_z(k) == 1) r = two::template load_at<dir_x(k)>(sb + k * S::SLOT + dir_y(k) * W, SEP);
                    else if constexpr (dir_z(k) == 0) r = c0[z_rank(k)];
                    else r = m1[z_rank(k)];
                    f[opp(k)] = two::widen(r);
                });
                cell_rule2<St>(f, lid, wall, ctx.inv_tau, ctx.lid_u);
                uint32_t ha = 0, hb = 0;
                if constexpr (St::stochastic) {
                    const uint32_t rh = sr_hash((uint32_t)g.ref(0, y, p - 1), step + 1);
                    ha = sr_cell(rh, xa);
                    hb = sr_cell(rh, xa + SEP);
                }
                // At a row's end the second cell is the wall behind it.  Predicated stores instead of a branch of
                // their own are 1-8 % faster (FP32; 16-bit, for rows that do not fill their warp), but not with the
                // dither of F16SR (2-4 % slower).
                // Stores of the default policy: the neighbours' parts of a sector meet in L2. Streaming ones were slower:
                // FP32 256^3 0.458 -> 0.450 ms a pair, batches of 64^3 0.750 -> 0.730 and of 40 x 72 x 50 0.531 -> 0.503
                // when it was changed.
                auto push = [&](auto cells) {
                    constexpr int kCells = decltype(cells)::value;  // 0: as vb says
                    static_for<0, Q>([&](auto kc) {
                        constexpr int k = decltype(kc)::value;
                        const raw r = two::narrow(f[k], ha, hb, k);
                        bits* const q = reinterpret_cast<bits*>(slots.push[k] + off);
                        const bool second = kCells == 0 ? vb : kCells == 2;
                        if constexpr (k16 && dir_x(k) == 0) {
                            if (second) *reinterpret_cast<raw*>(q) = r;
                            else *q = two::first(r);
                        } else {
                            *q = two::first(r);
                            if (second) q[SEP] = two::second(r);
                        }
                    });
                };
                using std::integral_constant;
                if (k16 && (St::stochastic ? vb : whole_rows)) push(integral_constant<int, 2>{});
                else push(integral_constant<int, St::stochastic ? 1 : 0>{});
            }
            // what beta pulls from this plane for the cells of this plane and of the next
            static_for<0, Q>([&](auto kc) {
                constexpr int k = decltype(kc)::value;
                if constexpr (dir_z(k) == 0) {
                    c0[z_rank(k)] = two::template load_at<dir_x(k)>(sb + k * S::SLOT + dir_y(k) * W, SEP);
                }
                if constexpr (dir_z(k) == -1) {
                    m1[z_rank(k)] = m2[z_rank(k)];
                    m2[z_rank(k)] = two::template load_at<dir_x(k)>(sb + k * S::SLOT + dir_y(k) * W, SEP);
                }
            });
        }
        named_arrive(1 + NST + stage, S::NB + 32);
        stage = stage + 1 == NST ? 0 : stage + 1;
    }
    named_arrive(1 + NST + stage, S::NB + 32);
}

template <class St, int TX, int TY, int NST, bool BATCH>
__global__ void __launch_bounds__(PairShape<St, TX, TY, NST, BATCH>::THREADS, 1)
    pair_step(const __grid_constant__ CUtensorMap map, const __grid_constant__ PairCtx one,
              const uint32_t* __restrict__ step_base, const uint32_t step_off, const PairWork w,
              int* __restrict__ err)
{
    using S = PairShape<St, TX, TY, NST, BATCH>;
    extern __shared__ __align__(128) unsigned char pair_smem[];
    __shared__ PairCtx many[BATCH ? kPairContexts : 1];
    auto* const smem = reinterpret_cast<typename St::bits*>(pair_smem);
    uint64_t* const full = reinterpret_cast<uint64_t*>(smem + NST * S::STAGE);
    int* const item_of = reinterpret_cast<int*>(full + NST);
    volatile int* const issued = item_of + NST;
    if (threadIdx.x == 0) {
        for (int s = 0; s < NST; ++s) {
            tma::mbar_init(&full[s], 1);
            issued[s] = 1;
        }
        tma::fence_mbar_init();
    }
    __syncthreads();
    allow_next_step();  // its blocks take the SMs that this one's leave
    const PairSource<St, TX, TY, BATCH> src{one, many};
    const uint32_t step = step_of<St>(step_base, step_off);
    if (threadIdx.x < S::NA) pair_alpha<St, TX, TY, NST, BATCH>(src, step, smem, full, item_of, issued, w.limit_ns, err);
    else if (threadIdx.x < S::NA + S::NB) pair_beta<St, TX, TY, NST, BATCH>(src, step, smem, item_of);
    else pair_copy<St, TX, TY, NST, BATCH>(&map, src, w, smem, full, item_of, issued);
}

}  // namespace lbm
