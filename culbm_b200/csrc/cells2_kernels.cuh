// Step kernels of the 16-bit formats on two neighbouring cells per thread,
// for even nx.
//
// One cell per thread, the 16-bit steps are bound by instruction issue: 612
// instructions per cell of the FP16-SR pull, against half the bytes of FP32.
// Two cells in one row share every address and, with even nx, an aligned
// 32-bit word of every plane, and their collision runs in packed FP32
// (packed2.cuh): 457 instructions per cell.  The pulled values stay in their
// stored form and are widened twice, once for the moments and once for the
// relaxation, and each pair of directions is narrowed and stored as soon as
// it is relaxed, so that the two cells run at 80 registers (six blocks of 128;
// at 128 registers the pull runs a fifth slower, at 64 it spills more).
// Threads take the pairs of a plane (in place: of its inner rows) in memory
// order, so warps are full whatever nx is.  Equilibrium cells (the row's ends
// of an inlet: a fifth of the warps at nx = 288) run with the fluid cells in
// the packed code.
//
// Each kernel comes in two codes.  The one for fluid issues all loads before
// the op bytes are looked at, and leaves walls and other cells to the one-cell
// code after it.  The one for mixed domains (mixed_domain, sim.cu) looks first
// and leaves the loads of idle pairs out; walls run along in the packed code,
// their stored values reversed, and a cell's half of a word is stored alone
// where the other cell is not packed.  256x256x160 FP16-SR, pull and in place,
// fluid code -> mixed code (one cell per thread): 60 % walls in blocks of 5^3
// cells 373 -> 239 us (283) and 444 -> 298 (326), seven eighths idle 131 -> 64
// (76) and 111 -> 71 (98).  One kernel with both codes runs fluid 7 % slower.
//
// FP16-SR channel with spheres, 288x272x280: pull 591 -> 476 us per step
// (46.1k MLUPS, 0.76 of the copy bandwidth), in place 663 -> 590 us; 512x512x256
// in place 1942 -> 1709 us.
//
// Odd nx keeps the one-cell kernels: without words the same code needs 108
// 16-bit accesses per pair instead of 72, and the load/store units then bound
// it (BF16-SR pull at 211x157x149: 138 us with pairs that straddle rows or
// lie 32 apart, 135 us one cell per thread).
#pragma once

#include <algorithm>

#include "packed2.cuh"
#include "stream_kernels.cuh"

namespace culbm {

constexpr int kCells2Threads = 128, kCells2Blocks = 6;

// Division of 0 <= n < 2^31 by a divisor fixed on the host, by Granlund and
// Montgomery's multiplication with the rounded-up reciprocal ("Division by
// invariant integers using multiplication", 1994); n + umulhi(n, m) stays
// below 2^32.
struct FastDiv {
    uint32_t m, s;
    __host__ void set(uint32_t d)
    {
        s = 0;
        while ((1ull << s) < d) ++s;
        m = static_cast<uint32_t>(((1ull << 32) * ((1ull << s) - d)) / d + 1);
    }
    __host__ __device__ __forceinline__ uint32_t div(uint32_t n) const
    {
        return (static_cast<uint32_t>((static_cast<uint64_t>(n) * m) >> 32) + n) >> s;
    }
};

// The two stored values of a word widened to their raw FP32 values.
template <typename S>
__device__ __forceinline__ f32x2 widen2(uint32_t w)
{
    if constexpr (ScaleExp<S>::value != 0) {
        const float2 v = __half22float2(*reinterpret_cast<const __half2*>(&w));
        return pk2(v.x, v.y);
    } else {
        return pk2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
    }
}

__device__ __forceinline__ uint32_t ld_word(const void* p)
{
    uint32_t v;
    asm volatile("ld.global.L2::256B.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ld_half(const void* p)
{
    unsigned short v;
    asm volatile("ld.global.L2::256B.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
// A value this thread has just stored (ordered after its stores).
__device__ __forceinline__ unsigned short ld_back(const void* p)
{
    unsigned short v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p) : "memory");
    return v;
}
// A pair of cells: index and position of cell 0 (x even; cell 1 is at x + 1),
// and whether cell 0 sits on the low x-face, cell 1 on the high one.
struct Pair {
    int i, x, y, z;
    bool lo, hi;
};

// The pair whose cell 0 is cell q of plane z.
__device__ __forceinline__ Pair pair_at(const Domain& D, const FastDiv& row, int q, int z)
{
    Pair c;
    c.y = static_cast<int>(row.div(static_cast<uint32_t>(q)));
    c.x = q - c.y * D.nx;
    c.z = z;
    c.i = q + D.nxy * z;
    c.lo = c.x == 0;
    c.hi = c.x + 2 == D.nx;
    return c;
}

// Cell k of a pair as the one-cell code takes it.
__device__ __forceinline__ CellCoord cell_in_pair(const Pair& c, int k)
{
    return {c.x + k, c.y, c.z, c.i + k, true};
}

// Cells of the packed code: plain fluid (LOAD, COLLIDE, STORE), equilibrium
// cells (EQU, STORE) and, in the code for mixed domains, walls (LOAD,
// bounce-back, STORE).
__device__ __forceinline__ bool op_fluid(uint32_t op) { return (op & 0x1Fu) == (OP_LOAD | OP_COLLIDE | OP_STORE); }
__device__ __forceinline__ bool op_equ(uint32_t op) { return (op & (0x1Fu ^ OP_LOAD)) == (OP_EQU | OP_STORE); }
__device__ __forceinline__ bool op_wall(uint32_t op) { return (op & 0x1Fu) == (OP_LOAD | OP_BB | OP_STORE); }

struct PairKind {
    bool e0, e1;    // cell 0, 1 is an equilibrium cell
    bool b0, b1;    // cell 0, 1 is a wall (mixed domains)
    bool p0, p1;    // cell 0, 1 goes through the packed code
    bool equ;       // some lane of the warp has an equilibrium cell
    bool wall;      // some lane of the warp has a wall (mixed domains)
    bool all;       // every cell of the warp's pairs goes through the packed code
};

// The votes are over whichever lanes arrive together: they choose between
// codes with the same results.
template <bool MIXED>
__device__ __forceinline__ PairKind pair_kind(uint32_t ops)
{
    PairKind k;
    k.e0 = op_equ(ops);
    k.e1 = op_equ(ops >> 8);
    k.b0 = MIXED && op_wall(ops);
    k.b1 = MIXED && op_wall(ops >> 8);
    k.p0 = k.e0 || k.b0 || op_fluid(ops);
    k.p1 = k.e1 || k.b1 || op_fluid(ops >> 8);
    const unsigned lanes = __activemask();
    k.equ = __any_sync(lanes, k.e0 || k.e1);
    k.wall = MIXED && __any_sync(lanes, k.b0 || k.b1);
    k.all = __all_sync(lanes, k.p0 && k.p1);
    return k;
}

// The macroscopic inputs of a warp's equilibrium cells on their way to L1
// while the populations load.
template <typename S>
__device__ __forceinline__ void prefetch_equ(const StepArgs<S, float>& a, const PairKind& k, int i)
{
    if (!(k.e0 || k.e1)) return;
    for (const float* p : {a.rho, a.vx, a.vy, a.vz}) asm volatile("prefetch.global.L1 [%0];" ::"l"(p + i));
}

// Update of two cells with pulled words w[d] (those of a cell outside the
// packed code are computed and unused): emit(k, p, q) takes the narrowed
// values of cell 0 (p) and cell 1 (q), direction k < 13 in bits 0-15 and
// 26 - k in bits 16-31 (k = 13: both in bits 0-15).  An equilibrium cell runs
// as a fluid cell with zero pulled values, its own rho and u, w = 1 and
// 1 - w = -0: -0 * 0 + feq is feq to the sign of a zero.
template <typename S, bool MIXED, class F>
__device__ __forceinline__ void relax_two(const StepArgs<S, float>& a, const PairKind& kind, int i, f32x2 z0,
                                          uint32_t* w, F&& emit)
{
    constexpr int E = ScaleExp<S>::value;
    const uint32_t h0 = IsSR<S>::value ? cell_hash(static_cast<uint32_t>(i), a.seed) : 0u;
    const uint32_t h1 = IsSR<S>::value ? cell_hash(static_cast<uint32_t>(i) + 1u, a.seed) : 0u;
    if (kind.equ) {
        const uint32_t keep = (kind.e0 ? 0u : 0xFFFFu) | (kind.e1 ? 0u : 0xFFFF0000u);
#pragma unroll
        for (int d = 0; d < 27; ++d) w[d] &= keep;
    }
    collide_fast2<E>(
        a.inv_tau, z0, [&](int d) { return widen2<S>(w[d]); },
        [&] {
            // the compiler would otherwise keep the 54 widened values
#pragma unroll
            for (int d = 0; d < 27; ++d) asm volatile("" : "+r"(w[d]));
        },
        [&](FastTerms2& t) {
            if (!kind.equ) return;
            const bool e0 = kind.e0, e1 = kind.e1;
            auto put = [&](f32x2& v, float x0, float x1) { v = pk2(e0 ? x0 : lo2(v), e1 ? x1 : hi2(v)); };
            const float r0 = e0 ? a.rho[i] : 1.0f, r1 = e1 ? a.rho[i + 1] : 1.0f;
            put(t.rho, r0, r1);
            put(t.dr, __fsub_rn(r0, 1.0f), __fsub_rn(r1, 1.0f));
            put(t.ux, e0 ? a.vx[i] : 0.0f, e1 ? a.vx[i + 1] : 0.0f);
            put(t.uy, e0 ? a.vy[i] : 0.0f, e1 ? a.vy[i + 1] : 0.0f);
            put(t.uz, e0 ? a.vz[i] : 0.0f, e1 ? a.vz[i + 1] : 0.0f);
            const float W[4] = {8.0f / 27.0f, 2.0f / 27.0f, 1.0f / 54.0f, 1.0f / 216.0f};
#pragma unroll
            for (int k = 0; k < 4; ++k) put(t.b[k], W[k] * pow2<float, E>(), W[k] * pow2<float, E>());
            put(t.om, -0.0f, -0.0f);
        },
        [&](int k, f32x2 fk, f32x2 fe) {
            uint32_t v0, v1;
            if (k < 13) {
                v0 = Pack2<S>::cvt(lo2(fe), lo2(fk), IsSR<S>::value ? sr_word_pair(h0, k) : 0u);
                v1 = Pack2<S>::cvt(hi2(fe), hi2(fk), IsSR<S>::value ? sr_word_pair(h1, k) : 0u);
            } else {
                v0 = enc16_raw<S>(lo2(fk), h0, 13);
                v1 = enc16_raw<S>(hi2(fk), h1, 13);
            }
            if (MIXED && kind.wall) {   // a wall's stored values as they are, reversed
                if (kind.b0) v0 = __byte_perm(w[26 - k], w[k], 0x5410);
                if (kind.b1) v1 = __byte_perm(w[26 - k], w[k], 0x7632);
            }
            emit(k, v0, v1);
        });
}

// The cells of a pair outside the packed code (done0, done1: not), through
// the one-cell code one(k): a round for a lane's first such cell, a round for
// its second.
template <class F>
__device__ __forceinline__ void other_cells(bool done0, bool done1, F&& one)
{
    if (done0 && done1) return;
    const int rounds = done0 || done1 ? 1 : 2;
#pragma unroll 1
    for (int k = done0 ? 1 : 0, r = 0; r < rounds; ++r, ++k) one(k);
}

// A cell that does not store changes nothing.
__device__ __forceinline__ bool op_keeps(uint32_t op) { return (op & OP_STORE) == 0; }

// Direction d of an emitted pair: its two values as one word, or one cell's value.
__device__ __forceinline__ uint32_t both_of(int d, uint32_t p, uint32_t q)
{
    return __byte_perm(p, q, d <= 13 ? 0x5410 : 0x7632);
}
__device__ __forceinline__ unsigned short one_of(int d, uint32_t v)
{
    return static_cast<unsigned short>(d <= 13 ? v : v >> 16);
}

template <typename S>
__device__ __forceinline__ void st_two(S* p, int d, uint32_t v0, uint32_t v1)
{
    *reinterpret_cast<uint32_t*>(p) = both_of(d, v0, v1);
}

// st_two for the cells of a pair that went through the packed code.
template <typename S>
__device__ __forceinline__ void st_packed(const PairKind& k, S* p, int d, uint32_t v0, uint32_t v1)
{
    if (k.all || (k.p0 && k.p1))
        st_two(p, d, v0, v1);
    else
        st16(p + (k.p1 ? 1 : 0), one_of(d, k.p1 ? v1 : v0));
}

// Whether a cell of the pair loads.
__device__ __forceinline__ bool pair_loads(uint32_t ops) { return (ops & (OP_LOAD | OP_LOAD << 8)) != 0; }

// Op bytes of a pair (cell 0 in bits 0-7).
__device__ __forceinline__ uint32_t ops_of(const uint8_t* ops, int i)
{
    return *reinterpret_cast<const unsigned short*>(ops + i);
}

// The pull step src -> dst of a pair.  An x-face cell pulls the directions
// whose source lies outside from its own column: the value the other cell of
// the pair pulls.  Its load past the row's side is not used; it stays inside
// the 27 planes (cx = +1 has d >= 2, cx = -1 has d <= 24).
template <bool MIXED, typename S>
__device__ __forceinline__ void pull_pair(const StepArgs<S, float>& a, const Pair& c, f32x2 nzero)
{
    const Domain& D = a.dom;
    const uint32_t ops = ops_of(a.ops, c.i);
    const int ym = c.y == 0 ? 0 : -D.nx, yp = c.y == D.ny - 1 ? 0 : D.nx;
    const int zm = c.z == 0 ? 0 : -D.nxy, zp = c.z == D.nz - 1 ? 0 : D.nxy;
    uint32_t w[27];   // not mixed: loaded before the op bytes are looked at
    if (!MIXED || pair_loads(ops)) {
#pragma unroll
        for (int d = 0; d < 27; ++d) {
            const int oy = cy_of(d) == 1 ? ym : cy_of(d) == -1 ? yp : 0;
            const int oz = cz_of(d) == 1 ? zm : cz_of(d) == -1 ? zp : 0;
            const S* p = a.src.p[d] + (c.i + oy + oz);
            if (cx_of(d) == 0) {
                w[d] = ld_word(p);
            } else {
                const uint32_t u = ld_half(p - cx_of(d)), v = ld_half(p + 1 - cx_of(d));
                w[d] = cx_of(d) == 1 ? __byte_perm(c.lo ? v : u, v, 0x5410) : __byte_perm(u, c.hi ? u : v, 0x5410);
            }
        }
    } else {
#pragma unroll
        for (int d = 0; d < 27; ++d) w[d] = 0;
    }
    const PairKind kind = pair_kind<MIXED>(ops);
    prefetch_equ(a, kind, c.i);
    auto one = [&](int k) { pull_cell<S, float>(a, cell_in_pair(c, k)); };
    if (MIXED) {
        if (kind.p0 || kind.p1)
            relax_two<S, MIXED>(a, kind, c.i, nzero, w, [&](int k, uint32_t v0, uint32_t v1) {
                st_packed(kind, a.dst.p[k] + c.i, k, v0, v1);
                if (k < 13) st_packed(kind, a.dst.p[26 - k] + c.i, 26 - k, v0, v1);
            });
        other_cells(kind.p0 || op_keeps(ops), kind.p1 || op_keeps(ops >> 8), one);
    } else {
        // the packed result of a cell outside the packed code is overwritten below; one without STORE keeps its slots
        const bool packed = (kind.p0 || kind.p1) && (ops & (ops >> 8) & OP_STORE);
        if (packed)
            relax_two<S, MIXED>(a, kind, c.i, nzero, w, [&](int k, uint32_t v0, uint32_t v1) {
                st_two(a.dst.p[k] + c.i, k, v0, v1);
                if (k < 13) st_two(a.dst.p[26 - k] + c.i, 26 - k, v0, v1);
            });
        // its halves are stored after the words, as another type: nothing may move between
        asm volatile("" ::: "memory");
        other_cells(kind.p0 && packed, kind.p1 && packed, one);
    }
}

// One pull step over the planes z0 + blockIdx.y.
template <typename S, bool MIXED>
__global__ void __launch_bounds__(kCells2Threads, kCells2Blocks)
    k_pull_cells2(const __grid_constant__ StepArgs<S, float> a, FastDiv row, int z0, f32x2 nzero)
{
    const Domain& D = a.dom;
    step_enter(a.overlap != 0);
    const uint32_t t = 2 * (blockIdx.x * kCells2Threads + threadIdx.x);   // cell 0 within the plane
    if (t >= static_cast<uint32_t>(D.nxy)) return;
    const Pair c = pair_at(D, row, static_cast<int>(t), z0 + static_cast<int>(blockIdx.y));
    pull_pair<MIXED>(a, c, nzero);
}

// Launch of an in-place step over the planes of a SlabSplit: first `faces`
// blocks that take the y/z-face rows one cell per thread (general clamp
// code), then `blocks_per_plane` blocks per interior plane for the pairs of
// its inner rows.  (Face blocks spread over the launch instead evict the inner
// rows' code from the instruction caches: 66.6 against 64.5 us per FP16-SR
// step at 160x120x100, 598 against 596 us at 288x272x280.)
struct Cells2Grid {
    SlabSplit q;
    FastDiv row, per_plane;
    int faces, blocks_per_plane;
};

inline Cells2Grid cells2_grid(const Domain& D, int za, int zb, long long* blocks)
{
    Cells2Grid g{};
    g.q = slab_split(D, za, zb);
    const long long face = 1ll * g.q.nzf * D.nxy + (D.ny > 1 ? 2ll : 1ll) * g.q.ni * D.nx;
    const long long inner = D.ny > 2 ? 1ll * D.nx * (D.ny - 2) : 0;   // even
    g.faces = static_cast<int>((face + kCells2Threads - 1) / kCells2Threads);
    g.blocks_per_plane = static_cast<int>((inner + 2 * kCells2Threads - 1) / (2 * kCells2Threads));
    *blocks = g.faces + 1ll * g.blocks_per_plane * g.q.ni;
    g.row.set(static_cast<uint32_t>(D.nx));
    g.per_plane.set(static_cast<uint32_t>(std::max(g.blocks_per_plane, 1)));
    return g;
}

// Face-row cell t of a launch (0-based over the slab's z-face planes, then
// its y-face rows).
__device__ __forceinline__ bool face_cell(const Domain& D, const Cells2Grid& g, uint32_t ut, CellCoord& c)
{
    const int zfaces = g.q.nzf * D.nxy;
    if (ut >= 0x80000000u) return false;
    const int t = static_cast<int>(ut);
    if (t < zfaces) {
        const int second = t >= D.nxy ? 1 : 0;
        const int r = t - second * D.nxy;
        c.y = static_cast<int>(g.row.div(static_cast<uint32_t>(r)));
        c.x = r - c.y * D.nx;
        c.z = (second == 0 && g.q.za == 0) ? 0 : D.nz - 1;
    } else {
        const int r = static_cast<int>(g.row.div(static_cast<uint32_t>(t - zfaces)));
        c.x = t - zfaces - r * D.nx;
        if (D.ny > 1) {
            if (r >= 2 * g.q.ni) return false;
            c.z = g.q.zlo + (r >> 1);
            c.y = (r & 1) ? D.ny - 1 : 0;
        } else {
            if (r >= g.q.ni) return false;
            c.z = g.q.zlo + r;
            c.y = 0;
        }
    }
    c.i = c.x + D.nx * (c.y + D.ny * c.z);
    c.valid = true;
    return true;
}

// This thread's pair of the inner rows, or false.
__device__ __forceinline__ bool inner_pair(const Domain& D, const Cells2Grid& g, uint32_t b, Pair& c)
{
    const uint32_t plane = g.per_plane.div(b);
    const uint32_t t = 2 * ((b - plane * g.blocks_per_plane) * kCells2Threads + threadIdx.x);
    if (t >= static_cast<uint32_t>(D.nx) * (D.ny - 2)) return false;
    c = pair_at(D, g.row, D.nx + static_cast<int>(t), g.q.zlo + static_cast<int>(plane));
    return true;
}

// Edge-buffer slot of a cell on an x-face for direction d (cx = +1: low face).
template <typename S>
__device__ __forceinline__ S* xface_slot(const StepArgs<S, float>& a, int d, int y, int z)
{
    return const_cast<S*>(xface_edge_ptr(a.edge, a.dom, a.el, cx_of(d) == 1 ? 0 : 1, d, y, z));
}

// In-place odd step (aa_odd_cell) of a pair in the inner rows.
template <bool MIXED, typename S>
__device__ __forceinline__ void aa_odd_pair(const StepArgs<S, float>& a, const Pair& c, f32x2 nzero)
{
    const Domain& D = a.dom;
    const uint32_t ops = ops_of(a.ops, c.i);
    uint32_t w[27];   // not mixed: loaded before the op bytes are looked at
    if (!MIXED || pair_loads(ops)) {
#pragma unroll
        for (int d = 0; d < 27; ++d) {
            const S* p = a.src.p[26 - d] + (c.i - nb_off(D, d));
            if (cx_of(d) == 0) {
                w[d] = ld_word(p);
            } else {
                // the value of a face cell whose source lies outside comes from the edge buffer below
                uint32_t u = 0, v = 0;
                if (!(cx_of(d) == 1 && c.lo)) u = ld_half(p);
                if (!(cx_of(d) == -1 && c.hi)) v = ld_half(p + 1);
                w[d] = __byte_perm(u, v, 0x5410);
            }
        }
    } else {
#pragma unroll
        for (int d = 0; d < 27; ++d) w[d] = 0;
    }
    const PairKind kind = pair_kind<MIXED>(ops);
    const bool f0 = kind.p0, f1 = kind.p1;
    if (f0 || f1) {
        prefetch_equ(a, kind, c.i);
        if (c.lo) {
#pragma unroll
            for (int d = 2; d < 27; d += 3) w[d] = __byte_perm(ld_half(xface_slot(a, d, c.y, c.z)), w[d], 0x7610);
        }
        if (c.hi) {
#pragma unroll
            for (int d = 0; d < 27; d += 3) w[d] = __byte_perm(w[d], ld_half(xface_slot(a, d, c.y, c.z)), 0x5410);
        }
        relax_two<S, MIXED>(a, kind, c.i, nzero, w, [&](int k, uint32_t v0, uint32_t v1) {
            auto out = [&](int d) {
                S* p = a.dst.p[d] + (c.i + nb_off(D, d));
                if (cx_of(d) == 0) {
                    st_packed(kind, p, d, v0, v1);
                    return;
                }
                // the streaming targets, except one outside the domain; a face cell is also the clamped source
                // of the cell on its own face
                const unsigned short s0 = one_of(d, v0), s1 = one_of(d, v1);
                if (f0 && !(cx_of(d) == -1 && c.lo)) st16(p, s0);
                if (f1 && !(cx_of(d) == 1 && c.hi)) st16(p + 1, s1);
                if (cx_of(d) == 1 && f0 && c.lo) st16(p - 1, s0);
                if (cx_of(d) == -1 && f1 && c.hi) st16(p + 2, s1);
            };
            out(k);
            if (k < 13) out(26 - k);
        });
    }
    other_cells(f0 || (MIXED && op_keeps(ops)), f1 || (MIXED && op_keeps(ops >> 8)), [&](int k) { aa_odd_cell<S, float, ROWS_INNER_ONE>(a, cell_in_pair(c, k)); });
}

template <typename S, bool MIXED>
__global__ void __launch_bounds__(kCells2Threads, kCells2Blocks)
    k_aa_odd_cells2(const __grid_constant__ StepArgs<S, float> a, const __grid_constant__ Cells2Grid g, f32x2 nzero)
{
    const Domain& D = a.dom;
    step_enter(a.overlap != 0);
    if (blockIdx.x < static_cast<uint32_t>(g.faces)) {
        CellCoord c;
        if (face_cell(D, g, blockIdx.x * kCells2Threads + threadIdx.x, c)) aa_odd_cell<S, float, ROWS_OUTER>(a, c);
        return;
    }
    Pair c;
    if (!inner_pair(D, g, blockIdx.x - static_cast<uint32_t>(g.faces), c)) return;
    aa_odd_pair<MIXED>(a, c, nzero);
}

// In-place even step (aa_even_cell) of a pair in the inner rows.
template <bool MIXED, typename S>
__device__ __forceinline__ void aa_even_pair(const StepArgs<S, float>& a, const Pair& c, f32x2 nzero)
{
    const uint32_t ops = ops_of(a.ops, c.i);
    uint32_t w[27];   // not mixed: loaded before the op bytes are looked at
    if (!MIXED || pair_loads(ops)) {
#pragma unroll
        for (int d = 0; d < 27; ++d) w[d] = ld_word(a.src.p[d] + c.i);
    } else {
#pragma unroll
        for (int d = 0; d < 27; ++d) w[d] = 0;
    }
    const PairKind kind = pair_kind<MIXED>(ops);
    const bool f0 = kind.p0, f1 = kind.p1;
    if (f0 || f1) {
        prefetch_equ(a, kind, c.i);
        relax_two<S, MIXED>(a, kind, c.i, nzero, w, [&](int k, uint32_t v0, uint32_t v1) {
            st_packed(kind, a.dst.p[26 - k] + c.i, k, v0, v1);
            if (k < 13) st_packed(kind, a.dst.p[k] + c.i, 26 - k, v0, v1);
        });
        // a face cell files f_d for the cell on its face whose clamped pull reads it: from the slots just written
        auto file = [&](int first, int k) {   // directions first, first + 3, ... (cx = +1: 2, cx = -1: 0)
#pragma unroll 1
            for (int d = first; d < 27; d += 3)
                st16(xface_slot(a, d, c.y + cy_of(d), c.z + cz_of(d)), ld_back(a.dst.p[26 - d] + (c.i + k)));
        };
        if (c.lo && f0) file(2, 0);
        if (c.hi && f1) file(0, 1);
    }
    other_cells(f0 || (MIXED && op_keeps(ops)), f1 || (MIXED && op_keeps(ops >> 8)), [&](int k) { aa_even_cell<S, float, ROWS_INNER>(a, cell_in_pair(c, k)); });
}

template <typename S, bool MIXED>
__global__ void __launch_bounds__(kCells2Threads, kCells2Blocks)
    k_aa_even_cells2(const __grid_constant__ StepArgs<S, float> a, const __grid_constant__ Cells2Grid g, f32x2 nzero)
{
    const Domain& D = a.dom;
    step_enter(a.overlap != 0);
    if (blockIdx.x < static_cast<uint32_t>(g.faces)) {
        CellCoord c;
        if (face_cell(D, g, blockIdx.x * kCells2Threads + threadIdx.x, c)) aa_even_cell<S, float, ROWS_OUTER>(a, c);
        return;
    }
    Pair c;
    if (!inner_pair(D, g, blockIdx.x - static_cast<uint32_t>(g.faces), c)) return;
    aa_even_pair<MIXED>(a, c, nzero);
}

}  // namespace culbm
