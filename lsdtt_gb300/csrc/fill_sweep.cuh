// fill_sweep.cuh -- one value window of the epsilon fill (fill_window.cuh)
// replayed by a whole thread block, one FIFO sweep at a time.
//
// A sweep is the reference's processing of the FIFO entries f_1..f_m present
// when the previous sweep ended, with the heap pops interleaved between them.
// Within a sweep every pop has a time T: the FIFO entry f_g pops at
// (g, 1); a heap cell of value k and index i pops at (g, 0, k, i), where g
// is its gap -- the first FIFO index at or after the moment it was queued
// whose value exceeds k (before f_g the heap pops everything below v_g, in
// value order). A cell queued before the sweep has gap NG(1, k); one that a
// pop discovers inherits the gap of its discoverer (the next gap after a
// FIFO entry), advanced to the next FIFO value above k. A cell not yet
// queued is discovered by the neighbour that pops first, i.e. with the
// smallest T, in that neighbour's direction order; it is raised (next
// sweep's FIFO, ordered by (T of the discoverer, direction)) when it is not
// above the discoverer's value, and otherwise queued as a heap cell (a pop
// of this sweep if its gap exists). Those rules define every T of the sweep
// as a fixed point, found in rounds: each round re-evaluates the cells next
// to the pops that changed in the previous one (a changed pop can only move
// the cells next to it). Between sweeps, when the FIFO runs empty, the block
// takes single heap pops by the sequential rules of win_replay.
//
// The replay is latency-bound (one sweep after another, each a few hundred
// cells), so a sweep takes the form with the shortest chain of dependent
// steps that holds it: short and narrow sweeps keep their pops and the cells
// they reach in shared memory and read one record per (pop, direction); wide
// ones keep one 16-byte event record per cell in global memory. With the wide
// form alone a 1500 x 1403 pitted fractal filled in 329 ms (21,705 sweeps)
// and a 256-member ensemble step took 241 ms; with the three, 163 and 186 ms
// (148 and 171 with what has changed around them since).
#pragma once

#include <cstdint>

#include "fill_window.cuh"

namespace lsdtt_gb300
{
namespace
{

constexpr int kSwThreads = 512;
// (the chain block has a whole SM to itself: its registers fill it, so the
// shared memory is sized to hold the widest FIFO generations of large basins)
constexpr int kSwFQ = 4096;  // FIFO entries of one sweep (a power of two)
constexpr int kSwL = 4096;   // entries of each per-sweep list (changed pops, discovered cells)
constexpr int kSwLv = 4;     // levels of the heap cells at or above the near threshold

// A cell's pop in the current sweep: valid when st is the sweep's id.
struct __align__(16) SwEv
{
    std::uint64_t hi;  // (gap << 33) | (kind << 32) | value key; kind 1 = FIFO entry
    std::uint32_t st;
    float val;
};

// A cell's discoverer in the current sweep (valid when te_st is the sweep's id).
struct __align__(16) SwTe
{
    std::uint64_t hi;   // discoverer's T
    std::uint32_t lo;   // its tie word (its cell for heap pops, 0 for FIFO entries)
    float val;          // its value
};

// Per-member scratch of the block replay (member-local, one entry per cell
// unless stated). Stamps make every array valid without clearing: a value
// counts only when it carries the current window's or sweep's id.
struct SweepBufs
{
    std::uint32_t* cst;      // state words of the records (WinGrid::rec[i].w at cst[4 i]): queued by window w = w + 2
    SwEv* ev;
    SwTe* te;
    std::uint32_t* te_st;    // sweep id: the discoverer in te is valid
    std::uint8_t* te_k;      // direction from the discoverer
    std::uint32_t* mk_c;     // round id: re-evaluated in this round (one thread per cell);
                             // a value at or below the sweep's id: not yet in this sweep
    std::uint32_t *dc, *dc2; // heap cells discovered earlier, not popped, with a value
    float *dk, *dk2;         //   below the threshold T ("near", two buffers)
    std::uint32_t* lc;       // the same at or above T, in kSwLv levels of lstride entries:
    float* lk;               //   level 0 below Lb[1], level k in [Lb[k], Lb[k+1]), the last
    std::size_t lstride;     //   unbounded; the bands grow 16-fold, a level is gathered and
                             //   spread again only when T reaches its lower bound (a radix heap)
    std::uint32_t* sc;       // spare list the gathering goes through
    float* sk;
};

// Scratch of a short sweep (sw_short): its pops and a table of the cells they
// reach (kWinNone / all ones between sweeps).
constexpr int kSwSM = 128;    // FIFO entries of a short sweep
constexpr int kSwSE = 512;    // its pops
constexpr int kSwSH = 2048;   // table entries
constexpr int kSwSC = 1536;   // cells in the table at most (three a thread)
struct SweepShort
{
    std::uint64_t key[kSwSH];  // least pop that reached the cell (sw_key | place << 3 | direction)
    std::uint64_t ek[kSwSE];   // time of a pop (sw_key)
    std::uint32_t cell[kSwSH];
    float z[kSwSH];            // its elevation
    std::uint32_t ec[kSwSE];
    std::uint16_t used[kSwSC];
    // counters of alternate sweeps, one in use while the other is reset:
    // pops; cells in the table; raised cells | near-list entries << 16
    std::uint32_t ne[2], nu[2], out[2], over;
};

// Scratch of a narrow sweep (sw_narrow): its pops ("events"), and every cell
// it touches in an open-addressing table. Entries of the table that are not
// in use hold kWinNone / kSwNoEv / 0 between sweeps.
constexpr int kSwNH = 4096;   // table entries (a power of two)
constexpr int kSwNE = 2048;   // cells in the table at most, hence also events and raised cells
constexpr int kSwNM = 1024;   // FIFO entries a narrow sweep takes on
constexpr int kSwProbe = 64;  // probes before the table counts as full
constexpr std::uint16_t kSwNoEv = 0xffffu;
struct SweepEvents
{
    std::uint64_t eh[kSwNE];   // event's time (sw_hi); all ones: withdrawn
    std::uint32_t ec[kSwNE];   // its cell
    float ev[kSwNE];           // its value
    std::uint32_t hk[kSwNH];   // cell
    float hz[kSwNH];           // its elevation (cells reached by a pop)
    std::uint32_t hd[kSwNH];   // discoverer: (event << 3) | direction
    std::uint32_t hm[kSwNH];   // (last round that touched it << 1) | look at all neighbours again
    std::uint16_t he[kSwNH];   // its own event
    std::uint16_t used[kSwNE], touched[kSwNE], la[kSwNE], lb[kSwNE];
    float pm[kSwNM];           // running maximum of the FIFO's values
};
struct SweepRaised
{
    std::uint64_t nhi[kSwNE];  // raised cells: discoverer's time, tie word and direction
    std::uint32_t nlo[kSwNE], nc[kSwNE];
    float nv[kSwNE];
    std::uint8_t nk[kSwNE];
    std::uint16_t idx[kSwNE];
};
struct SweepNarrow : SweepEvents, SweepRaised
{
};

// Scratch of a wide sweep.
struct SweepWide
{
    std::uint16_t ng[kSwFQ + 2];
    std::uint32_t nc[kSwFQ];
    float nv[kSwFQ];
    std::uint64_t nhi[kSwFQ];
    std::uint32_t nlo[kSwFQ];
    std::uint8_t nk[kSwFQ];
    std::uint32_t la[kSwL], lb[kSwL], lt[kSwL];
};

static_assert(sizeof(SweepShort) <= sizeof(SweepEvents), "the short form leaves the raised cells' arrays alone");

struct SweepShared
{
    std::uint32_t fc[kSwFQ];
    alignas(16) float fv[kSwFQ];
    union
    {
        SweepNarrow n;
        SweepShort t;  // over n's SweepEvents
        SweepWide w;
    };
    std::uint32_t cnt[12];
    float red_v[kSwThreads / 32];
    std::uint32_t red_i[kSwThreads / 32];
    std::uint32_t red_s[kSwThreads / 32];
    std::int64_t red_p;
};

__device__ __forceinline__ std::uint64_t sw_hi(std::uint32_t g, std::uint32_t kind, float key)
{
    return (static_cast<std::uint64_t>(g) << 33) | (static_cast<std::uint64_t>(kind) << 32) | float_order_key(key);
}

// FIFOs up to this length are searched entry by entry; longer ones through
// the next-greater table ng
constexpr std::uint32_t kSwScan = 64;

// A cell's record, read as memory holds it now: the block writes state words
// into the records while it reads them, so these loads must not take the
// read-only path that the compiler may choose for a pointer to const.
__device__ __forceinline__ float4 sw_record(const float4* p)
{
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}

// first FIFO index >= g0 (1-based) whose value exceeds key; m + 1 if none
__device__ __forceinline__ std::uint32_t sw_ng(const SweepShared& sh, std::uint32_t m, std::uint32_t g0, float key)
{
    // (an event read while its cell's thread writes it can pair the sweep's
    // stamp with a time of zero: gap 0, whose table entry does not exist and
    // sent the search round for ever. The writer lists the cell, so the round
    // after reads it whole.)
    std::uint32_t g = max(g0, 1u);
    if (m <= kSwScan)
        while (g <= m && !(sh.fv[g - 1] > key)) ++g;
    else
        while (g <= m && !(sh.fv[g - 1] > key)) g = sh.w.ng[g];
    return g;
}

// ---- narrow sweeps ---------------------------------------------------------
// A sweep whose cells fit the shared-memory table (a FIFO generation of up to
// about a thousand entries; LEM surfaces and most sweeps of a pitted fractal
// hold about ten to a hundred with their few hundred heap pops). The wide form
// below re-evaluates every not-yet-queued cell next to a changed pop by
// loading the event records of its eight neighbours from global memory, once
// for every pop that reaches it: about 16,000 scattered 16-byte loads a sweep
// of 180 pops, bound by the L1's tag rate and by the latency of its dependent
// steps, 14-17 us. Here a pop instead pushes itself to its eight neighbours:
// one record load per (pop, direction) says whether the cell is open, and the
// cell's discoverer is the least pop pushed to it, kept in the table. Only a
// pop whose time moved after it was pushed, or that was withdrawn, makes its
// neighbours look at all of theirs again (in the table). The fixed point is
// the same one: each cell's time follows from strictly earlier pops.

// Counters of one narrow sweep.
struct SwNarrowCtl
{
    std::uint32_t ne, used, over1, over2, nf, vkey;
    std::uint32_t touched[2], next[2];
};

// One position of the sorted list per thread, kept across sweeps.
struct SwList
{
    std::int64_t base;
    float4 o;
    __device__ void load(const WinGrid& G, int tid)
    {
        o = base + tid < G.nsorted ? G.ordRec[base + tid] : make_float4(INFINITY, INFINITY, 0.0f, 0.0f);
    }
};

__device__ void sw_narrow_clear(SweepNarrow& n)
{
    for (int k = threadIdx.x; k < kSwNH; k += kSwThreads)
    {
        n.hk[k] = kWinNone;
        n.hd[k] = kWinNone;
        n.hm[k] = 0u;
        n.he[k] = kSwNoEv;
    }
}

// Table position of `cell`, entered if new (*fresh); -1: the table is full.
__device__ __forceinline__ int sw_insert(SweepNarrow& n, std::uint32_t cell, bool* fresh)
{
    std::uint32_t h = (cell * 2654435761u) >> 20;
    for (int p = 0; p < kSwProbe; ++p)
    {
        const std::uint32_t prev = atomicCAS(&n.hk[h], kWinNone, cell);
        if (prev == kWinNone)
        {
            *fresh = true;
            return static_cast<int>(h);
        }
        if (prev == cell) return static_cast<int>(h);
        h = (h + 1) & (kSwNH - 1);
    }
    return -1;
}

__device__ __forceinline__ int sw_find(const SweepNarrow& n, std::uint32_t cell)
{
    std::uint32_t h = (cell * 2654435761u) >> 20;
    for (int p = 0; p < kSwProbe; ++p)
    {
        const std::uint32_t k = n.hk[h];
        if (k == cell) return static_cast<int>(h);
        if (k == kWinNone) return -1;
        h = (h + 1) & (kSwNH - 1);
    }
    return -1;
}

// Tie word of an event's time: its cell for heap pops, 0 for FIFO entries.
__device__ __forceinline__ std::uint32_t sw_lo(const SweepNarrow& n, std::uint32_t e, std::uint64_t hi)
{
    return ((hi >> 32) & 1u) ? 0u : n.ec[e];
}

// Does discoverer a = (event << 3) | direction come before b?
__device__ __forceinline__ bool sw_before(const SweepNarrow& n, std::uint32_t a, std::uint32_t b)
{
    if (b == kWinNone) return true;
    const std::uint32_t ea = a >> 3, eb = b >> 3;
    if (ea == eb) return (a & 7u) < (b & 7u);
    const std::uint64_t ha = n.eh[ea], hb = n.eh[eb];
    if (ha != hb) return ha < hb;
    return sw_lo(n, ea, ha) < sw_lo(n, eb, hb);
}

// First FIFO index >= g0 (1-based) whose value exceeds key; m + 1 if none.
// Where nothing before g0 exceeds it either, the running maximum is searched.
__device__ __forceinline__ std::uint32_t sw_gap(const SweepShared& sh, std::uint32_t m, std::uint32_t g0, float key)
{
    if (g0 > m) return m + 1;
    if (g0 > 1 && sh.n.pm[g0 - 2] > key)
    {
        std::uint32_t g = g0;
        while (g <= m && !(sh.fv[g - 1] > key)) ++g;
        return g;
    }
    std::uint32_t lo = g0, hi = m + 1;
    while (lo < hi)
    {
        const std::uint32_t mid = (lo + hi) >> 1;
        if (sh.n.pm[mid - 1] > key) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// The raised cells nc/nv[0 .. mn) into fc/fv in push order: by the
// discoverer's time, tie word and direction (distinct keys). Up to 128, L
// threads count the entries before one (L = 512 / mn rounded up to a power of
// two), past that a bitonic sort of indices. One thread per entry took 5,000
// of a sweep's 21,000 cycles at 40 entries.
__device__ __forceinline__ void sw_rank(SweepShared& sh, std::uint32_t mn)
{
    SweepNarrow& n = sh.n;
    const int tid = threadIdx.x;
    if (mn <= 128)
    {
        int lg = 5;
        while ((mn << lg) > static_cast<std::uint32_t>(kSwThreads)) --lg;
        const std::uint32_t a = static_cast<std::uint32_t>(tid) >> lg, l = tid & ((1u << lg) - 1u);
        const bool in = a < mn;
        std::uint32_t rank = 0;
        if (in)
        {
            const std::uint64_t ah = n.nhi[a];
            for (std::uint32_t b = l; b < mn; b += 1u << lg)
            {
                const std::uint64_t bh = n.nhi[b];
                if (bh < ah)
                    ++rank;
                else if (bh == ah && b != a &&
                         (n.nlo[b] < n.nlo[a] || (n.nlo[b] == n.nlo[a] && n.nk[b] < n.nk[a])))
                    ++rank;
            }
        }
        for (int o = (1 << lg) >> 1; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
        if (in && l == 0)
        {
            sh.fc[rank] = n.nc[a];
            sh.fv[rank] = n.nv[a];
        }
        return;
    }
    const std::uint32_t P = 1u << (32 - __clz(mn - 1));
    for (std::uint32_t t = tid; t < P; t += kSwThreads) n.idx[t] = static_cast<std::uint16_t>(t);
    __syncthreads();
    auto after = [&](std::uint32_t a, std::uint32_t b) {
        if (a >= mn) return b < mn || a > b;
        if (b >= mn) return false;
        if (n.nhi[a] != n.nhi[b]) return n.nhi[a] > n.nhi[b];
        if (n.nlo[a] != n.nlo[b]) return n.nlo[a] > n.nlo[b];
        return n.nk[a] > n.nk[b];
    };
    for (std::uint32_t k = 2; k <= P; k <<= 1)
        for (std::uint32_t j = k >> 1; j > 0; j >>= 1)
        {
            for (std::uint32_t i = tid; i < P; i += kSwThreads)
            {
                const std::uint32_t l = i ^ j;
                if (l > i)
                {
                    const std::uint32_t a = n.idx[i], b = n.idx[l];
                    if (after(a, b) == ((i & k) == 0))
                    {
                        n.idx[i] = static_cast<std::uint16_t>(b);
                        n.idx[l] = static_cast<std::uint16_t>(a);
                    }
                }
            }
            __syncthreads();
        }
    for (std::uint32_t r = tid; r < mn; r += kSwThreads)
    {
        const std::uint32_t a = n.idx[r];
        sh.fc[r] = n.nc[a];
        sh.fv[r] = n.nv[a];
    }
}

// ---- short sweeps ----------------------------------------------------------
// Most sweeps are far smaller than the narrow form's room: 39 FIFO entries, 28
// heap pops and 146 cells reached on average on a 1500 x 1403 pitted fractal,
// 10, 69 and 158 on a 256-member LEM ensemble, and one or two rounds settle
// them. Such a sweep is a chain of dependent steps with hardly any work in
// them, so this form keeps only what the chain needs: a pop's time and place
// pack into one 64-bit word, so one atomic minimum finds a cell's discoverer,
// a word shows whether a cell has to be settled again, and the heap cells
// below T are read ahead during the sweep before. A sweep that does not fit,
// or in which a pop would move after it was pushed, is left to the narrow
// form; nothing but the spare lists has been written by then.

// Time of a pop as one word: gap, kind (1 FIFO entry), value key; the low
// seven bits are left for the discoverer's place among the cell's neighbours
// (its tie word: their row-major order) and the direction to the cell.
__device__ __forceinline__ std::uint64_t sw_key(std::uint32_t g, std::uint32_t kind, float v)
{
    return (static_cast<std::uint64_t>(g) << 40) | (static_cast<std::uint64_t>(kind) << 39) |
           (static_cast<std::uint64_t>(kind ? 0u : float_order_key(v)) << 7);
}

// First FIFO index >= g0 (1-based, g0 >= 1) whose value exceeds key, m + 1 if
// none, sixteen entries at a time (m <= kSwSM; fv is 16-byte aligned).
__device__ __forceinline__ std::uint32_t sw_gap_short(const SweepShared& sh, std::uint32_t m, std::uint32_t g0, float key)
{
    for (std::uint32_t b = (g0 - 1) & ~15u; b < m; b += 16)
    {
        std::uint32_t above = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            const float4 v = *reinterpret_cast<const float4*>(sh.fv + b + 4 * k);
            above |= (v.x > key ? 1u : 0u) << (4 * k);
            above |= (v.y > key ? 2u : 0u) << (4 * k);
            above |= (v.z > key ? 4u : 0u) << (4 * k);
            above |= (v.w > key ? 8u : 0u) << (4 * k);
        }
        if (b < g0 - 1) above &= 0xffffu << (g0 - 1 - b);
        if (m - b < 16) above &= (1u << (m - b)) - 1u;
        if (above) return b + __ffs(above);
    }
    return m + 1;
}

// Near-list entries read ahead: entry tid of the current list.
struct SwNear
{
    std::uint32_t c;
    float k;
    bool ok;  // block-uniform
};

template <class Open, class Lvc, class Lvk, class Level>
__device__ bool sw_short(const WinGrid& G, const SweepBufs& B, SweepShared& sh, SwList& lst, SwNear& near,
                         const Open& open_rec, float S, std::uint32_t wst, std::uint32_t m, std::uint32_t q, float Vmax,
                         float T, std::int64_t& s_p, std::uint32_t& s_nd, const std::uint32_t* dc, const float* dk,
                         std::uint32_t* dc2, float* dk2, const Lvc& lvc, const Lvk& lvk, std::uint32_t* s_nl,
                         const Level& level_of, float* out_F, float& s_V, std::uint32_t& s_m)
{
    SweepShort& t = sh.t;
    const int tid = threadIdx.x, lane = tid & 31;
    const float inv_nc = 1.0f / static_cast<float>(G.nc);
    // a warp's share of a shared counter (all lanes call it)
    auto claim = [&](bool want, std::uint32_t* ctr) -> std::uint32_t {
        const unsigned b = __ballot_sync(0xffffffffu, want);
        if (!b) return 0u;
        const int lead = __ffs(b) - 1;
        std::uint32_t base = 0;
        if (lane == lead) base = atomicAdd(ctr, static_cast<std::uint32_t>(__popc(b)));
        return __shfl_sync(0xffffffffu, base, lead) + __popc(b & ((1u << lane) - 1u));
    };
    auto heap_pop = [&](bool want, std::uint32_t c, float key) {
        const std::uint32_t e = claim(want, &t.ne[q]);
        if (want && e < static_cast<std::uint32_t>(kSwSE))
        {
            t.ek[e] = sw_key(sw_gap_short(sh, m, 1, key), 0, key);
            t.ec[e] = c;
        }
    };
    // ---- the pops ----
    std::uint32_t own_c = 0;
    float own_v = 0.0f;
    if (static_cast<std::uint32_t>(tid) < m)
    {
        own_c = sh.fc[tid];
        own_v = sh.fv[tid];
        t.ek[tid] = sw_key(tid + 1, 1, 0.0f);
        t.ec[tid] = own_c;
    }
    const std::uint32_t nd = s_nd;
    if (nd)
    {
        const bool in = static_cast<std::uint32_t>(tid) < nd;
        if (!near.ok && in)
        {
            near.c = dc[tid];
            near.k = dk[tid];
        }
        const bool pops = in && near.k < Vmax;
        heap_pop(pops, near.c, near.k);
        // the rest stay (counted in the high half)
        const unsigned b = __ballot_sync(0xffffffffu, in && !pops);
        if (b)
        {
            const int lead = __ffs(b) - 1;
            std::uint32_t base = 0;
            if (lane == lead) base = atomicAdd(&t.out[q], static_cast<std::uint32_t>(__popc(b)) << 16);
            const std::uint32_t k =
                (__shfl_sync(0xffffffffu, base, lead) >> 16) + __popc(b & ((1u << lane) - 1u));
            if (in && !pops)
            {
                dc2[k] = near.c;
                dk2[k] = near.k;
            }
        }
    }
    std::int64_t p = s_p;
    if (p < lst.base || p >= lst.base + kSwThreads)
    {
        lst.base = p;
        lst.load(G, tid);
    }
    std::uint32_t ne;
    for (;;)
    {
        const bool below = lst.base + tid < G.nsorted && lst.o.x < Vmax;
        heap_pop(below && lst.base + tid >= p && lst.o.y < S, __float_as_uint(lst.o.z), lst.o.x);
        const int cnt = __syncthreads_count(below);
        ne = t.ne[q];
        if (lst.base + cnt > p) p = lst.base + cnt;
        if (cnt < kSwThreads) break;
        __syncthreads();  // every thread has read the count before it grows
        if (ne > static_cast<std::uint32_t>(kSwSE)) return false;
        lst.base += kSwThreads;
        lst.load(G, tid);
    }
    if (ne > static_cast<std::uint32_t>(kSwSE)) return false;
    // ---- rounds ----
    // Phase 1 pushes the new pops to their open neighbours; in phase 2 thread
    // i settles cells i, i + 512, ... of the table again where a lesser pop
    // has reached them, and those that pop in this sweep are the next round's
    // new pops. A pop that would move or be withdrawn after it was pushed is
    // left to the narrow form.
    constexpr int kV = kSwSC / kSwThreads;
    const int dir = tid & 7;
    const unsigned lower = (1u << lane) - 1u;
    std::uint64_t last[kV], pop[kV];  // the key a cell was last settled with; its time if it pops (else 0)
    int what[kV];                     // 1 raised, 2 heap cell below T, 3 heap cell at or above it, 4 pops
    std::uint32_t hv[kV], jv[kV];     // its place in the table, and the cell
    float zv[kV];
#pragma unroll
    for (int v = 0; v < kV; ++v)
    {
        last[v] = ~0ull;
        pop[v] = 0;
        what[v] = 0;
    }
    std::uint32_t e0 = 0, e1 = ne, nu = 0;
    for (int round = 0;; ++round)
    {
        for (std::uint32_t i0 = e0 * 8; i0 < e1 * 8; i0 += 3 * kSwThreads)
        {
            int rs[3], cs[3];
            float4 rc[3];
            bool ok[3];
#pragma unroll
            for (int u = 0; u < 3; ++u)
            {
                const std::uint32_t i = i0 + u * kSwThreads + tid;
                ok[u] = false;
                if (i < e1 * 8)
                {
                    const std::uint32_t c = t.ec[i >> 3];
                    const int r0 = win_row(c, G.nc, inv_nc);
                    const int c0 = static_cast<int>(c - static_cast<std::uint32_t>(r0) * G.nc);
                    ok[u] = fill_nb(G.nr, G.nc, G.per_ns, G.per_ew, r0, c0, dir, rs[u], cs[u]);
                    if (ok[u]) rc[u] = sw_record(G.rec + (static_cast<std::uint32_t>(rs[u]) * G.nc + cs[u]));
                }
            }
            int fresh[3];
            std::uint32_t before = 0, all = 0;
#pragma unroll
            for (int u = 0; u < 3; ++u)
            {
                fresh[u] = -1;
                if (ok[u] && open_rec(rc[u]))
                {
                    const int r = rs[u], c = cs[u];
                    const std::uint32_t j = static_cast<std::uint32_t>(r) * G.nc + c;
                    // the pop's place among the neighbours of the cell, in
                    // row-major order of their indices (an axis that wraps
                    // reorders its ends)
                    int pr = 1 - d8_dr(dir), pc = 1 - d8_dc(dir);
                    if (G.per_ns && (r == 0 || r == G.nr - 1))
                    {
                        const int r0 = r - d8_dr(dir) < 0 ? G.nr - 1 : (r - d8_dr(dir) >= G.nr ? 0 : r - d8_dr(dir));
                        const int up = r == 0 ? G.nr - 1 : r - 1, dn = r == G.nr - 1 ? 0 : r + 1;
                        pr = (up < r0) + (r < r0) + (dn < r0);
                    }
                    if (G.per_ew && (c == 0 || c == G.nc - 1))
                    {
                        const int c0 = c - d8_dc(dir) < 0 ? G.nc - 1 : (c - d8_dc(dir) >= G.nc ? 0 : c - d8_dc(dir));
                        const int le = c == 0 ? G.nc - 1 : c - 1, ri = c == G.nc - 1 ? 0 : c + 1;
                        pc = (le < c0) + (c < c0) + (ri < c0);
                    }
                    const std::uint64_t key = t.ek[(i0 + u * kSwThreads + tid) >> 3] |
                                              static_cast<std::uint64_t>((3 * pr + pc) << 3 | dir);
                    std::uint32_t h = (j * 2654435761u) >> 21;
                    int probe = 0;
                    for (; probe < 32; ++probe)
                    {
                        const std::uint32_t prev = atomicCAS(&t.cell[h], kWinNone, j);
                        if (prev == kWinNone)
                        {
                            fresh[u] = static_cast<int>(h);
                            t.z[h] = rc[u].x;
                            break;
                        }
                        if (prev == j) break;
                        h = (h + 1) & (kSwSH - 1);
                    }
                    if (probe < 32)
                        atomicMin(reinterpret_cast<unsigned long long*>(&t.key[h]),
                                  static_cast<unsigned long long>(key));
                    else t.over = 1;
                }
                const unsigned b = __ballot_sync(0xffffffffu, fresh[u] >= 0);
                before += __popc(b & lower);
                all += __popc(b);
            }
            if (all)
            {
                std::uint32_t base = 0;
                if (lane == 0) base = atomicAdd(&t.nu[q], all);
                std::uint32_t k = __shfl_sync(0xffffffffu, base, 0) + before;
#pragma unroll
                for (int u = 0; u < 3; ++u)
                    if (fresh[u] >= 0)
                    {
                        if (k < static_cast<std::uint32_t>(kSwSC)) t.used[k] = static_cast<std::uint16_t>(fresh[u]);
                        ++k;
                    }
            }
        }
        __syncthreads();
        nu = t.nu[q];
        if (t.over || nu > static_cast<std::uint32_t>(kSwSC)) return false;
        if (tid == 0 && round == 0) t.out[q ^ 1u] = t.nu[q ^ 1u] = 0;
        bool moved = false;
#pragma unroll
        for (int v = 0; v < kV; ++v)
        {
            if (static_cast<std::uint32_t>(v) * kSwThreads >= nu) break;  // (block-uniform)
            const std::uint32_t i = v * kSwThreads + tid;
            std::uint64_t np = 0;
            if (i < nu)
            {
                if (!what[v])
                {
                    hv[v] = t.used[i];
                    jv[v] = t.cell[hv[v]];
                    zv[v] = t.z[hv[v]];
                }
                const std::uint64_t kd = t.key[hv[v]];
                if (kd != last[v])
                {
                    last[v] = kd;
                    const float z = zv[v];
                    const std::uint32_t gap = static_cast<std::uint32_t>(kd >> 40);
                    const std::uint32_t kind = static_cast<std::uint32_t>(kd >> 39) & 1u;
                    const float bval = kind ? sh.fv[gap - 1] : float_from_order_key(static_cast<std::uint32_t>(kd >> 7));
                    if (z <= bval) what[v] = 1;
                    else
                    {
                        what[v] = z < T ? 2 : 3;
                        if (z < Vmax)
                        {
                            const std::uint32_t g = sw_gap_short(sh, m, gap + kind, z);
                            if (g <= m)
                            {
                                what[v] = 4;
                                np = sw_key(g, 0, z);
                            }
                        }
                    }
                    if (pop[v] && np != pop[v]) moved = true;
                    if (np == pop[v]) np = 0;  // known already
                    else pop[v] = np;
                }
            }
            const std::uint32_t e = claim(np != 0, &t.ne[q]);
            if (np != 0 && e < static_cast<std::uint32_t>(kSwSE))
            {
                t.ek[e] = np;
                t.ec[e] = jv[v];
            }
        }
        if (__syncthreads_or(moved)) return false;
        e0 = e1;
        e1 = t.ne[q];
        if (e1 > static_cast<std::uint32_t>(kSwSE) || round == 30) return false;
        if (e1 == e0) break;
    }
    // ---- settled: raised and near cells, then the next generation ----
    std::uint32_t n1 = 0, n2 = 0, all = 0;
#pragma unroll
    for (int v = 0; v < kV; ++v)
    {
        const unsigned b1 = __ballot_sync(0xffffffffu, what[v] == 1), b2 = __ballot_sync(0xffffffffu, what[v] == 2);
        n1 += __popc(b1 & lower);
        n2 += __popc(b2 & lower);
        all += __popc(b1) + (static_cast<std::uint32_t>(__popc(b2)) << 16);
    }
    std::uint32_t k1 = 0, k2 = 0;
    if (all)
    {
        std::uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&t.out[q], all);
        base = __shfl_sync(0xffffffffu, base, 0);
        k1 = (base & 0xffffu) + n1;
        k2 = (base >> 16) + n2;
    }
#pragma unroll
    for (int v = 0; v < kV; ++v)
    {
        if (!what[v]) continue;
        const std::uint32_t h = hv[v], j = jv[v];
        if (what[v] == 1)
        {
            const std::uint64_t kd = last[v];
            const std::uint32_t gap = static_cast<std::uint32_t>(kd >> 40);
            const int d = static_cast<int>(kd & 7u);
            std::uint32_t lo = 0;
            float bval;
            if ((kd >> 39) & 1u) bval = sh.fv[gap - 1];
            else
            {
                bval = float_from_order_key(static_cast<std::uint32_t>(kd >> 7));
                // the discoverer's cell
                const int r = win_row(j, G.nc, inv_nc);
                const int c = static_cast<int>(j - static_cast<std::uint32_t>(r) * G.nc);
                int r0, c0;
                fill_nb(G.nr, G.nc, G.per_ns, G.per_ew, r, c, (d + 4) & 7, r0, c0);
                lo = static_cast<std::uint32_t>(r0) * G.nc + c0;
            }
            sh.n.nc[k1] = j;
            sh.n.nv[k1] = raise_from(bval, G.eps, (d & 1) ? G.Ld : G.L);
            sh.n.nhi[k1] = kd >> 7;
            sh.n.nlo[k1] = lo;
            sh.n.nk[k1] = static_cast<std::uint8_t>(d);
            ++k1;
        }
        else if (what[v] == 2)
        {
            dc2[k2] = j;
            dk2[k2] = zv[v];
            ++k2;
        }
        else if (what[v] == 3)
        {
            const float z = zv[v];
            const int lv = level_of(z);
            const std::uint32_t kl = s_nl[lv] + atomicAdd(&sh.cnt[7 + lv], 1u);
            lvc(lv)[kl] = j;
            lvk(lv)[kl] = z;
        }
        B.cst[4 * static_cast<std::size_t>(j)] = wst;
        t.cell[h] = kWinNone;
        t.key[h] = ~0ull;
    }
    if (static_cast<std::uint32_t>(tid) < m) out_F[own_c] = own_v;
    __syncthreads();
    const std::uint32_t mn = t.out[q] & 0xffffu, nn = t.out[q] >> 16;
    near.ok = nn <= static_cast<std::uint32_t>(kSwThreads);
    if (static_cast<std::uint32_t>(tid) < nn)
    {
        near.c = dc2[tid];
        near.k = dk2[tid];
    }
    if (tid == 0)
    {
        s_V = fmaxf(s_V, Vmax);
        s_nd = nn;
        for (int k = 0; k < kSwLv; ++k) s_nl[k] += sh.cnt[7 + k];
        s_p = p;
        s_m = mn;
        t.ne[q ^ 1u] = mn;
    }
    sw_rank(sh, mn);
    __syncthreads();
    return true;
}

// One narrow sweep of the FIFO fc/fv[0 .. m) by the whole block; pm and an
// empty table given. On success the next generation is in fc/fv, its length
// in s_m, and true is returned. Nothing outside shared memory and the spare
// near list (dc2, dk2) is written before it is certain that the sweep fits:
// false leaves it to the wide form.
template <class Open, class Lvc, class Lvk, class Level>
__device__ bool sw_narrow(const WinGrid& G, const SweepBufs& B, SweepShared& sh, SwNarrowCtl& C, SwList& lst,
                          const Open& open_rec, float S, std::uint32_t wst, std::uint32_t m, float Vmax, float T,
                          std::int64_t& s_p, std::uint32_t& s_nd, const std::uint32_t* dc, const float* dk,
                          std::uint32_t* dc2, float* dk2, const Lvc& lvc, const Lvk& lvk, std::uint32_t* s_nl,
                          const Level& level_of, float* out_F, float& s_V, std::uint32_t& s_m, std::uint32_t& s_mlim)
{
    SweepNarrow& n = sh.n;
    const int tid = threadIdx.x, lane = tid & 31;
    const float inv_nc = 1.0f / static_cast<float>(G.nc);
    const std::uint32_t nd = s_nd;
    // warp-wide append of `v` to a list; every lane of the warp calls it
    auto append = [&](bool want, std::uint16_t* list, std::uint32_t* ctr, std::uint32_t v, std::uint32_t* over) {
        const unsigned b = __ballot_sync(0xffffffffu, want);
        if (!b) return;
        const int lead = __ffs(b) - 1;
        std::uint32_t base = 0;
        if (lane == lead) base = atomicAdd(ctr, static_cast<std::uint32_t>(__popc(b)));
        base = __shfl_sync(0xffffffffu, base, lead);
        if (want)
        {
            const std::uint32_t k = base + __popc(b & ((1u << lane) - 1u));
            if (k < static_cast<std::uint32_t>(kSwNE)) list[k] = static_cast<std::uint16_t>(v);
            else *over = 1;
        }
    };
    // ---- the pops known beforehand ----
    auto enter = [&](bool want, std::uint32_t e, std::uint64_t hi, std::uint32_t c, float v) {
        bool fresh = false;
        int h = -1;
        if (want)
        {
            n.eh[e] = hi;
            n.ec[e] = c;
            n.ev[e] = v;
            n.la[e] = static_cast<std::uint16_t>(e);
            h = sw_insert(n, c, &fresh);
            if (h < 0) C.over1 = 1;
            else n.he[h] = static_cast<std::uint16_t>(e);
        }
        append(fresh, n.used, &C.used, static_cast<std::uint32_t>(h), &C.over1);
    };
    // a heap cell's event, numbered warp-wide
    auto enter_heap = [&](bool want, std::uint32_t c, float key) {
        const unsigned b = __ballot_sync(0xffffffffu, want);
        if (!b) return;
        const int lead = __ffs(b) - 1;
        std::uint32_t base = 0;
        if (lane == lead) base = atomicAdd(&C.ne, static_cast<std::uint32_t>(__popc(b)));
        base = __shfl_sync(0xffffffffu, base, lead);
        std::uint32_t e = base + __popc(b & ((1u << lane) - 1u));
        if (want && e >= static_cast<std::uint32_t>(kSwNE))
        {
            C.over1 = 1;
            want = false;
        }
        enter(want, e, want ? sw_hi(sw_gap(sh, m, 1, key), 0, key) : 0ull, c, key);
    };
    for (std::uint32_t g0 = 0; g0 < m; g0 += kSwThreads)
    {
        const std::uint32_t g = g0 + tid;
        const bool in = g < m;
        enter(in, g, sw_hi(g + 1, 1, 0.0f), in ? sh.fc[g] : 0u, in ? sh.fv[g] : 0.0f);
    }
    // heap cells discovered earlier: below Vmax they pop, the rest stay
    for (std::uint32_t t0 = 0; t0 < nd; t0 += kSwThreads)
    {
        const std::uint32_t t = t0 + tid;
        const bool in = t < nd;
        const std::uint32_t c = in ? dc[t] : 0u;
        const float key = in ? dk[t] : INFINITY;
        const bool pops = in && key < Vmax;
        enter_heap(pops, c, key);
        const bool keep = in && !pops;
        const unsigned b = __ballot_sync(0xffffffffu, keep);
        if (b)
        {
            const int lead = __ffs(b) - 1;
            std::uint32_t base = 0;
            if (lane == lead) base = atomicAdd(&sh.cnt[3], static_cast<std::uint32_t>(__popc(b)));
            base = __shfl_sync(0xffffffffu, base, lead);
            if (keep)
            {
                const std::uint32_t k = base + __popc(b & ((1u << lane) - 1u));
                dc2[k] = c;
                dk2[k] = key;
            }
        }
    }
    // the sorted list from s_p on: the values below Vmax come first, so
    // counting them gives the next position
    std::int64_t p = s_p;
    if (p < lst.base || p >= lst.base + kSwThreads)
    {
        lst.base = p;
        lst.load(G, tid);
    }
    for (;;)
    {
        const bool below = lst.base + tid < G.nsorted && lst.o.x < Vmax;
        enter_heap(below && lst.base + tid >= p && lst.o.y < S, __float_as_uint(lst.o.z), lst.o.x);
        const int cnt = __syncthreads_count(below);
        if (lst.base + cnt > p) p = lst.base + cnt;
        if (cnt < kSwThreads) break;
        if (__syncthreads_or(C.over1 != 0)) return false;
        lst.base += kSwThreads;
        lst.load(G, tid);
    }
    // ---- rounds ----
    // Phase 1 pushes the changed pops to their open neighbours; phase 2
    // re-evaluates the cells touched. Each flag and counter is written in one
    // phase and read in the other, so every thread sees the same value.
    std::uint32_t ne = min(C.ne, static_cast<std::uint32_t>(kSwNE)), nch = ne;
    std::uint16_t *la = n.la, *lb = n.lb;
    for (std::uint32_t round = 1;; ++round)
    {
        const std::uint32_t par = round & 1u;
        constexpr int kU = 3;
        for (std::uint32_t t0 = 0; t0 < nch * 8; t0 += kSwThreads * kU)
        {
            std::uint32_t ent[kU], js[kU];
            float4 q[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u)
            {
                const std::uint32_t t = t0 + u * kSwThreads + tid;
                js[u] = kWinNone;
                if (t < nch * 8)
                {
                    ent[u] = la[t >> 3];
                    const std::uint32_t c = n.ec[ent[u] & 0x7fffu];
                    const int r0 = win_row(c, G.nc, inv_nc);
                    const int c0 = static_cast<int>(c - static_cast<std::uint32_t>(r0) * G.nc);
                    int rr, cc;
                    if (fill_nb(G.nr, G.nc, G.per_ns, G.per_ew, r0, c0, static_cast<int>(t & 7), rr, cc))
                    {
                        js[u] = static_cast<std::uint32_t>(rr) * G.nc + cc;
                        q[u] = sw_record(G.rec + js[u]);
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < kU; ++u)
            {
                bool fresh = false, first = false;
                int h = -1;
                if (js[u] != kWinNone && open_rec(q[u]))
                {
                    h = sw_insert(n, js[u], &fresh);
                    if (h < 0) C.over1 = 1;
                    else
                    {
                        n.hz[h] = q[u].x;
                        const std::uint32_t moved = ent[u] >> 15;
                        if (!moved)
                        {
                            const std::uint32_t mine = (ent[u] << 3) | (tid & 7u);
                            std::uint32_t cur = *reinterpret_cast<volatile std::uint32_t*>(&n.hd[h]);
                            while (sw_before(n, mine, cur))
                            {
                                const std::uint32_t prev = atomicCAS(&n.hd[h], cur, mine);
                                if (prev == cur) break;
                                cur = prev;
                            }
                        }
                        first = (atomicMax(&n.hm[h], 2u * round + moved) >> 1) < round;
                    }
                }
                append(fresh, n.used, &C.used, static_cast<std::uint32_t>(h), &C.over1);
                append(first, n.touched, &C.touched[par], static_cast<std::uint32_t>(h), &C.over1);
            }
        }
        __syncthreads();
        if (C.over1) return false;
        const std::uint32_t nt = C.touched[par];
        if (tid == 0) C.touched[par ^ 1u] = C.next[par ^ 1u] = 0;
        for (std::uint32_t t0 = 0; t0 < nt; t0 += kSwThreads)
        {
            const std::uint32_t t = t0 + tid;
            bool born = false, changed = false;
            std::uint32_t h = 0, e = 0;
            std::uint64_t nh = ~0ull;
            float z = 0.0f;
            if (t < nt)
            {
                h = n.touched[t];
                z = n.hz[h];
                if (n.hm[h] & 1u)
                {
                    // the least pop among all of its neighbours (those born
                    // in this phase push themselves in the next round)
                    const std::uint32_t jc = n.hk[h];
                    const int r0 = win_row(jc, G.nc, inv_nc);
                    const int c0 = static_cast<int>(jc - static_cast<std::uint32_t>(r0) * G.nc);
                    std::uint32_t best = kWinNone;
                    for (int d = 0; d < 8; ++d)
                    {
                        int rr, cc;
                        if (!fill_nb(G.nr, G.nc, G.per_ns, G.per_ew, r0, c0, d, rr, cc)) continue;
                        const int pos = sw_find(n, static_cast<std::uint32_t>(rr) * G.nc + cc);
                        if (pos < 0) continue;
                        const std::uint32_t e2 = *reinterpret_cast<volatile std::uint16_t*>(&n.he[pos]);
                        if (e2 >= ne || n.eh[e2] == ~0ull) continue;
                        const std::uint32_t cand = (e2 << 3) | static_cast<std::uint32_t>((d + 4) & 7);
                        if (sw_before(n, cand, best)) best = cand;
                    }
                    n.hd[h] = best;
                }
                const std::uint32_t d = n.hd[h];
                e = n.he[h];
                if (d != kWinNone)
                {
                    const std::uint64_t bh = n.eh[d >> 3];
                    if (bh != ~0ull && !(z <= n.ev[d >> 3]))
                    {
                        const std::uint32_t gd = static_cast<std::uint32_t>(bh >> 33);
                        const std::uint32_t g = sw_gap(sh, m, ((bh >> 32) & 1u) ? gd + 1 : gd, z);
                        if (g <= m) nh = sw_hi(g, 0, z);
                    }
                }
                if (e == kSwNoEv) born = nh != ~0ull;
                else if (n.eh[e] != nh)
                {
                    n.eh[e] = nh;  // moved, withdrawn or back again
                    changed = true;
                }
            }
            const unsigned b = __ballot_sync(0xffffffffu, born);
            if (b)
            {
                const int lead = __ffs(b) - 1;
                std::uint32_t base = 0;
                if (lane == lead) base = atomicAdd(&C.ne, static_cast<std::uint32_t>(__popc(b)));
                base = __shfl_sync(0xffffffffu, base, lead);
                if (born)
                {
                    e = base + __popc(b & ((1u << lane) - 1u));
                    if (e < static_cast<std::uint32_t>(kSwNE))
                    {
                        n.eh[e] = nh;
                        n.ec[e] = n.hk[h];
                        n.ev[e] = z;
                        n.he[h] = static_cast<std::uint16_t>(e);
                    }
                    else C.over2 = 1;
                }
            }
            append(born || changed, lb, &C.next[par], changed ? e | 0x8000u : e, &C.over2);
        }
        __syncthreads();
        if (C.over2 || round == 60) return false;
        nch = C.next[par];
        ne = C.ne;
        if (nch == 0) break;
        std::uint16_t* t = la;
        la = lb;
        lb = t;
    }
    // ---- the sweep is settled: pops, next generation, heap cells ----
    for (std::uint32_t g = tid; g < m; g += kSwThreads) out_F[sh.fc[g]] = sh.fv[g];
    const std::uint32_t nu = C.used;
    for (std::uint32_t t0 = 0; t0 < nu; t0 += kSwThreads)
    {
        const std::uint32_t t = t0 + tid;
        bool raised = false;
        std::uint32_t j = 0, e = 0, dir = 0;
        float vpop = -INFINITY;
        if (t < nu)
        {
            const std::uint32_t h = n.used[t], d = n.hd[h], own = n.he[h];
            j = n.hk[h];
            const float z = n.hz[h];
            n.hk[h] = kWinNone;
            n.hd[h] = kWinNone;
            n.hm[h] = 0u;
            n.he[h] = kSwNoEv;
            if (d != kWinNone)
            {
                e = d >> 3;
                dir = d & 7u;
                if (own != kSwNoEv && n.eh[own] != ~0ull) vpop = z;
                else if (z <= n.ev[e]) raised = true;
                else if (z < T)
                {
                    const std::uint32_t k = atomicAdd(&sh.cnt[3], 1u);
                    dc2[k] = j;
                    dk2[k] = z;
                }
                else
                {
                    const int lv = level_of(z);
                    const std::uint32_t k = s_nl[lv] + atomicAdd(&sh.cnt[7 + lv], 1u);
                    lvc(lv)[k] = j;
                    lvk(lv)[k] = z;
                }
                B.cst[4 * static_cast<std::size_t>(j)] = wst;
            }
        }
        const unsigned b = __ballot_sync(0xffffffffu, raised);
        if (b)
        {
            const int lead = __ffs(b) - 1;
            std::uint32_t base = 0;
            if (lane == lead) base = atomicAdd(&C.nf, static_cast<std::uint32_t>(__popc(b)));
            base = __shfl_sync(0xffffffffu, base, lead);
            if (raised)
            {
                const std::uint32_t k = base + __popc(b & ((1u << lane) - 1u));
                const std::uint64_t hi = n.eh[e];
                n.nc[k] = j;
                n.nv[k] = raise_from(n.ev[e], G.eps, (dir & 1u) ? G.Ld : G.L);
                n.nhi[k] = hi;
                n.nlo[k] = sw_lo(n, e, hi);
                n.nk[k] = static_cast<std::uint8_t>(dir);
            }
        }
        for (int o = 16; o > 0; o >>= 1) vpop = fmaxf(vpop, __shfl_down_sync(0xffffffffu, vpop, o));
        if (lane == 0 && vpop > Vmax) atomicMax(&C.vkey, float_order_key(vpop));
    }
    __syncthreads();
    const std::uint32_t mn = C.nf;
    if (tid == 0)
    {
        s_V = fmaxf(fmaxf(s_V, Vmax), C.vkey ? float_from_order_key(C.vkey) : Vmax);
        s_nd = sh.cnt[3];
        for (int k = 0; k < kSwLv; ++k) s_nl[k] += sh.cnt[7 + k];
        s_p = p;
        s_m = mn;
        s_mlim = min(static_cast<std::uint32_t>(kSwNM), s_mlim + s_mlim / 8 + 1);
    }
    sw_rank(sh, mn);
    __syncthreads();
    return true;
}

// First k in [lo, n) with a(k) above the searched value (`above`, monotone in
// k; n if none), by one full warp: 32 probes a step, where one thread's
// bisection took a dependent load per halving (21 of them at 2 M cells).
template <class I, class Above>
__device__ __forceinline__ I sw_search(I lo, I n, const Above& above)
{
    const int lane = threadIdx.x & 31;
    I hi = n;
    while (hi - lo > 32)
    {
        const I step = (hi - lo + 31) / 32;
        const I k = lo + static_cast<I>(lane) * step;
        const unsigned b = __ballot_sync(0xffffffffu, k >= hi || above(k));
        const int f = b ? __ffs(b) - 1 : 32;
        const I top = lo + static_cast<I>(f) * step;
        if (f > 0) lo = lo + static_cast<I>(f - 1) * step + 1;
        hi = f == 0 ? lo : (top < hi ? top : hi);
    }
    const I k = lo + lane;
    const unsigned b = __ballot_sync(0xffffffffu, k >= hi || above(k));
    return b ? lo + static_cast<I>(__ffs(b) - 1) : hi;
}

// Block replay of window w (every thread of a kSwThreads block calls it).
// *ctr is the member's id counter (stamps), advanced here. Returns kWinOk
// with *next set, or kWinOverflow (a sweep's FIFO or lists above their
// shared-memory size, or no fixed point within its round limit) -- then
// nothing of the window is final and the caller replays it by the
// sequential rules.
__device__ int win_sweep_replay(const WinGrid& G, int w, const SweepBufs& B, float* out_F, std::uint32_t* ctr,
                                SweepShared& sh, int* next)
{
    const int tid = threadIdx.x;
    const float S = G.cuts[w];
    __shared__ std::uint32_t s_ctr, s_m, s_nd, s_sweep, s_status, s_last_move, s_mlim;
    __shared__ SwNarrowCtl s_nar;
    __shared__ std::uint32_t s_nl[kSwLv];
    __shared__ std::int64_t s_p;
    __shared__ float s_V, s_T, s_D;
    __shared__ float s_Lb[kSwLv];
    __shared__ int s_j;
    __shared__ int s_cnext, s_next, s_stop;
    __shared__ unsigned long long s_first;
    __shared__ float s_lz;
    __shared__ std::uint32_t s_lc;
    if (tid < 32)
    {
        const std::int64_t p =
            sw_search<std::int64_t>(0, G.nsorted, [&](std::int64_t k) { return !(G.ordRec[k].x < S); });
        if (tid == 0) s_p = p;
    }
    if (tid == 0)
    {
        s_ctr = *ctr;
        s_V = S;
        s_cnext = w + 1;
        s_m = 0;
        s_nd = 0;
        // near threshold T: four diagonal raise steps above the start
        // (adapted as the window goes); level bounds 16, 256, 4096 bands on
        s_D = fmaxf(4.0f * G.eps * G.Ld, 1e-6f * fabsf(S) + 1e-30f);
        s_T = S + s_D;
        float wb = 16.0f * s_D;
        s_Lb[0] = s_T;
        for (int k = 0; k < kSwLv; ++k) s_nl[k] = 0;
        for (int k = 1; k < kSwLv; ++k)
        {
            s_Lb[k] = s_T + wb;
            wb *= 16.0f;
        }
        s_last_move = 0;
        s_mlim = kSwNM;
        s_status = kWinOk;
        s_next = G.ncut;
        s_stop = 0;
    }
    __syncthreads();
    bool clean = false;  // the narrow table is empty (block-uniform)
    bool ready = false;  // the short table is empty and its counters are set (block-uniform)
    std::uint32_t q = 0;  // parity of the short sweeps' counters
    SwNear near{0, 0.0f, false};
    // (a wrapped axis one or two cells across reaches a cell twice)
    const bool short_ok = !((G.per_ns && G.nr <= 2) || (G.per_ew && G.nc <= 2));
    int short_rest = 0, short_back = 0;  // sweeps to go without trying the short form, after it gave up
    SwList lst;          // block of the sorted list, one position per thread
    lst.base = s_p;
    lst.load(G, tid);
    // not queued yet: valid, not popped before the window, not queued at its
    // start, not queued by this window (its state word)
    const std::uint32_t wst = static_cast<std::uint32_t>(w) + 2u;
    auto open_rec = [&](const float4& q) -> bool {
        const std::uint32_t st = __float_as_uint(q.w);
        return st != 0u && st != wst && q.y >= S && !(q.z < S);
    };
    auto open_cell = [&](std::uint32_t j, float& zj) -> bool {
        const float4 q = sw_record(G.rec + j);
        zj = q.x;
        return open_rec(q);
    };
    auto set_queued = [&](std::uint32_t j) { B.cst[4 * static_cast<std::size_t>(j)] = wst; };
    std::uint32_t* dc = B.dc;
    std::uint32_t* dc2 = B.dc2;
    float* dk = B.dk;
    float* dk2 = B.dk2;
    // level of a heap cell's key at or above T
    auto level_of = [&](float key) -> int {
        int k = 0;
        while (k + 1 < kSwLv && !(key < s_Lb[k + 1])) ++k;
        return k;
    };
    auto lvc = [&](int k) { return B.lc + static_cast<std::size_t>(k) * B.lstride; };
    auto lvk = [&](int k) { return B.lk + static_cast<std::size_t>(k) * B.lstride; };
    // a pass pops one cell (a background pop) or its sweep's FIFO, each cell
    // at most once, so more pops than cells means the replay has gone wrong:
    // it is then left to the sequential rules
    const std::uint64_t pass_cap = static_cast<std::uint64_t>(G.nr) * static_cast<std::uint64_t>(G.nc) + 2;
    std::uint64_t passes = 0;
    for (;;)
    {
        passes += max(s_m, 1u);
        if (passes > pass_cap)
        {
            if (tid == 0) s_status = kWinOverflow;
            __syncthreads();
            break;
        }
        if (s_m == 0)
        {
            // ---- FIFO empty: one heap pop by the sequential rules ----
            // (the list's head found 512 positions at a time, the cuts by a
            // warp, the neighbours a lane each: one thread doing all of it
            // took 28,000 cycles)
            if (tid == 0)
            {
                s_first = ~0ull;
                s_lc = kWinNone;
            }
            if (s_p < lst.base || s_p >= lst.base + kSwThreads)
            {
                lst.base = s_p;
                lst.load(G, tid);
            }
            __syncthreads();
            for (;;)
            {
                const std::int64_t q0 = lst.base + tid;
                const bool head = q0 >= s_p && q0 < G.nsorted && lst.o.y < S;
                const unsigned hb = __ballot_sync(0xffffffffu, head);
                if (head && static_cast<int>(tid & 31) == __ffs(hb) - 1)
                    atomicMin(&s_first, static_cast<unsigned long long>(q0));
                const bool more = lst.base + kSwThreads < G.nsorted;
                if (__syncthreads_or(head) || !more) break;
                lst.base += kSwThreads;
                lst.load(G, tid);
            }
            if (s_first == static_cast<unsigned long long>(lst.base + tid))
            {
                s_lz = lst.o.x;
                s_lc = __float_as_uint(lst.o.z);
            }
            // the least discovered heap cell: in the first non-empty list
            // (every near key is below T, and every level's keys below the
            // next level's)
            int which = -1;
            if (!s_nd)
            {
                which = kSwLv - 1;
                for (int k = kSwLv - 2; k >= 0; --k)
                    if (s_nl[k]) which = k;
            }
            const std::uint32_t* lc = which < 0 ? dc : lvc(which);
            const float* lk = which < 0 ? dk : lvk(which);
            const std::uint32_t ln = which < 0 ? s_nd : s_nl[which];
            float bz = INFINITY;
            std::uint32_t bi = kWinNone, bslot = kWinNone;
            for (std::uint32_t t = tid; t < ln; t += kSwThreads)
                if (win_key_less(lk[t], lc[t], bz, bi))
                {
                    bz = lk[t];
                    bi = lc[t];
                    bslot = t;
                }
            for (int o = 16; o > 0; o >>= 1)
            {
                const float oz = __shfl_down_sync(0xffffffffu, bz, o);
                const std::uint32_t oi = __shfl_down_sync(0xffffffffu, bi, o);
                const std::uint32_t os = __shfl_down_sync(0xffffffffu, bslot, o);
                if (win_key_less(oz, oi, bz, bi))
                {
                    bz = oz;
                    bi = oi;
                    bslot = os;
                }
            }
            if ((tid & 31) == 0)
            {
                sh.red_v[tid >> 5] = bz;
                sh.red_i[tid >> 5] = bi;
                sh.red_s[tid >> 5] = bslot;
            }
            __syncthreads();
            if (tid < 32)
            {
                const int lane = tid;
                bz = lane < kSwThreads / 32 ? sh.red_v[lane] : INFINITY;
                bi = lane < kSwThreads / 32 ? sh.red_i[lane] : kWinNone;
                bslot = lane < kSwThreads / 32 ? sh.red_s[lane] : kWinNone;
                for (int o = 16; o > 0; o >>= 1)
                {
                    const float oz = __shfl_xor_sync(0xffffffffu, bz, o);
                    const std::uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    const std::uint32_t os = __shfl_xor_sync(0xffffffffu, bslot, o);
                    if (win_key_less(oz, oi, bz, bi))
                    {
                        bz = oz;
                        bi = oi;
                        bslot = os;
                    }
                }
                const bool have_l = s_lc != kWinNone;
                float hz = have_l ? s_lz : INFINITY;
                std::uint32_t hc = s_lc;
                bool from_list = have_l;
                if (bi != kWinNone && (!have_l || win_key_less(bz, bi, hz, hc)))
                {
                    hz = bz;
                    hc = bi;
                    from_list = false;
                }
                const std::int64_t p = have_l ? static_cast<std::int64_t>(s_first) : G.nsorted;
                float V = s_V;
                int cn = s_cnext;
                bool stop = hc == kWinNone;
                if (stop) cn = G.ncut;
                else
                {
                    // first cut above V (sweeps leave it to this point)
                    cn = sw_search<int>(cn, G.ncut, [&](int k) { return G.cuts[k] > V; });
                    const bool trig = hz <= V && cn > 0 && G.cuts[cn - 1] >= hz;
                    stop = !trig && (cn >= G.ncut || G.cand[cn]);
                }
                if (lane == 0)
                {
                    s_p = (!stop && from_list) ? p + 1 : p;
                    if (stop)
                    {
                        s_next = cn;
                        s_stop = 1;
                    }
                }
                if (!stop)
                {
                    // the pop's open neighbours, a lane each
                    const int r = win_row(hc, G.nc, 1.0f / static_cast<float>(G.nc));
                    const int c = static_cast<int>(hc - static_cast<std::uint32_t>(r) * G.nc);
                    std::uint32_t j = kWinNone;
                    float zj = 0.0f;
                    int rr, cc;
                    if (lane < 8 && fill_nb(G.nr, G.nc, G.per_ns, G.per_ew, r, c, lane, rr, cc))
                    {
                        j = static_cast<std::uint32_t>(rr) * G.nc + cc;
                        if (!open_cell(j, zj)) j = kWinNone;
                    }
                    // (a cell reached twice across a short wrapped axis counts once)
                    for (int k = 0; k < 7; ++k)
                    {
                        const std::uint32_t other = __shfl_sync(0xffffffffu, j, k);
                        if (lane > k && j != kWinNone && other == j) j = kWinNone;
                    }
                    const bool raised = j != kWinNone && zj <= hz;
                    const int lv = (j == kWinNone || raised) ? -2 : (zj < s_T ? -1 : level_of(zj));
                    const unsigned rb = __ballot_sync(0xffffffffu, raised);
                    const unsigned lower = (1u << lane) - 1u;
                    // the popped heap cell leaves its list: the last entry takes its place
                    if (lane == 0 && !from_list)
                    {
                        if (which < 0)
                        {
                            const std::uint32_t last = --s_nd;
                            dc[bslot] = dc[last];
                            dk[bslot] = dk[last];
                        }
                        else
                        {
                            const std::uint32_t last = --s_nl[which];
                            std::uint32_t* wc = lvc(which);
                            float* wk = lvk(which);
                            wc[bslot] = wc[last];
                            wk[bslot] = wk[last];
                        }
                    }
                    __syncwarp();
                    if (raised)
                    {
                        const std::uint32_t m = __popc(rb & lower);
                        sh.fc[m] = j;
                        sh.fv[m] = raise_from(hz, G.eps, (lane & 1) ? G.Ld : G.L);
                    }
                    for (int k = -1; k < kSwLv; ++k)
                    {
                        const unsigned b = __ballot_sync(0xffffffffu, lv == k);
                        if (!b) continue;
                        std::uint32_t* ctr = k < 0 ? &s_nd : &s_nl[k];
                        const std::uint32_t at = *ctr + __popc(b & lower);
                        if (lv == k)
                        {
                            (k < 0 ? dc : lvc(k))[at] = j;
                            (k < 0 ? dk : lvk(k))[at] = zj;
                        }
                        __syncwarp();
                        if (lane == 0) *ctr += __popc(b);
                        __syncwarp();
                    }
                    if (j != kWinNone) set_queued(j);
                    if (lane == 0)
                    {
                        s_cnext = cn;
                        s_V = fmaxf(V, hz);
                        s_m = __popc(rb);
                    }
                }
            }
            __syncthreads();
            near.ok = ready = false;
            if (s_stop) break;
            continue;
        }
        // ---- one sweep ----
        const std::uint32_t m = s_m;
        const float T0 = s_T;
        if (tid == 0)
        {
            // the sweep's id, then ids for its rounds (sweep + 1 .. sweep + 64)
            s_sweep = ++s_ctr;
            s_ctr += 64;
            // cnt: [0] changed (la), [1] changed next (lb), [2] discovered
            // (lt), [3] surviving heap cells, [4] next FIFO, [5] overflow,
            // [6..10] moves and appends to the near list and the levels
            for (int k = 0; k < 12; ++k) sh.cnt[k] = 0;
        }
        // the FIFO's largest value: a short one every warp for itself
        float Vmax = -INFINITY;
        if (m <= static_cast<std::uint32_t>(kSwSM))
        {
            const std::uint32_t l = tid & 31;
#pragma unroll
            for (std::uint32_t g = 0; g < static_cast<std::uint32_t>(kSwSM); g += 32)
                if (g + l < m) Vmax = fmaxf(Vmax, sh.fv[g + l]);
            for (int o = 16; o > 0; o >>= 1) Vmax = fmaxf(Vmax, __shfl_xor_sync(0xffffffffu, Vmax, o));
        }
        else
        {
            for (std::uint32_t g = tid; g < m; g += kSwThreads) Vmax = fmaxf(Vmax, sh.fv[g]);
            for (int o = 16; o > 0; o >>= 1) Vmax = fmaxf(Vmax, __shfl_xor_sync(0xffffffffu, Vmax, o));
            if ((tid & 31) == 0) sh.red_v[tid >> 5] = Vmax;
            __syncthreads();
            Vmax = sh.red_v[0];
            for (int k = 1; k < kSwThreads / 32; ++k) Vmax = fmaxf(Vmax, sh.red_v[k]);
        }
        if (Vmax >= T0)
        {
            // the FIFO reaches T: raise it; the levels whose lower bound it
            // has reached (0 .. j) are gathered and spread again, below T to
            // the near list, the rest under new bounds (kept below level
            // j + 1's); each cell goes down a level at a time
            near.ok = false;
            __syncthreads();  // every thread has read T before it moves
            if (tid == 0)
            {
                const std::uint32_t sweep = s_sweep;
                // T moved again within 4 sweeps: widen the band; not within
                // 64: narrow it (a sweep's id advances by 65)
                if (sweep - s_last_move < 4u * 65u) s_D *= 2.0f;
                else if (sweep - s_last_move > 64u * 65u) s_D *= 0.5f;
                s_last_move = sweep;
                s_T = Vmax + s_D;
                s_Lb[0] = s_T;
                int jl = 0;
                for (int k = 1; k < kSwLv; ++k)
                    if (!(s_T < s_Lb[k])) jl = k;
                if (jl > 0)
                {
                    const float cap = jl + 1 < kSwLv ? s_Lb[jl + 1] : INFINITY;
                    float wb = 16.0f * s_D;
                    for (int k = 1; k <= jl; ++k)
                    {
                        s_Lb[k] = fminf(s_T + wb, cap);
                        wb *= 16.0f;
                    }
                }
                s_j = jl;
                for (int k = 6; k < 12; ++k) sh.cnt[k] = 0;
            }
            __syncthreads();
            const int jl = s_j;
            std::uint32_t ng_all = 0;
            for (int k = 0; k <= jl; ++k)
            {
                const std::uint32_t nk = s_nl[k];
                const std::uint32_t* src_c = lvc(k);
                const float* src_k = lvk(k);
                for (std::uint32_t t = tid; t < nk; t += kSwThreads)
                {
                    B.sc[ng_all + t] = src_c[t];
                    B.sk[ng_all + t] = src_k[t];
                }
                ng_all += nk;
            }
            __syncthreads();
            const float T = s_T;
            const std::uint32_t nd0 = s_nd;
            const int lane = tid & 31;
            auto warp_append = [&](bool want, std::uint32_t* dst_c, float* dst_k, std::uint32_t* ctr, std::uint32_t c,
                                   float key) {
                const unsigned b = __ballot_sync(0xffffffffu, want);
                if (!b) return;
                const int lead = __ffs(b) - 1;
                std::uint32_t base = 0;
                if (lane == lead) base = atomicAdd(ctr, static_cast<std::uint32_t>(__popc(b)));
                base = __shfl_sync(0xffffffffu, base, lead);
                if (want)
                {
                    const std::uint32_t k2 = base + __popc(b & ((1u << lane) - 1u));
                    dst_c[k2] = c;
                    dst_k[k2] = key;
                }
            };
            for (std::uint32_t t0 = 0; t0 < ng_all; t0 += kSwThreads)
            {
                const std::uint32_t t = t0 + tid;
                const bool in = t < ng_all;
                const std::uint32_t c = in ? B.sc[t] : 0u;
                const float key = in ? B.sk[t] : INFINITY;
                const int dest = !in ? -2 : (key < T ? -1 : level_of(key));
                warp_append(dest == -1, dc + nd0, dk + nd0, &sh.cnt[6], c, key);
                for (int k = 0; k <= jl; ++k) warp_append(dest == k, lvc(k), lvk(k), &sh.cnt[7 + k], c, key);
            }
            __syncthreads();
            if (tid == 0)
            {
                s_nd = nd0 + sh.cnt[6];
                for (int k = 0; k <= jl; ++k) s_nl[k] = sh.cnt[7 + k];
                for (int k = 0; k < 12; ++k) sh.cnt[k] = 0;
            }
            __syncthreads();
        }
        if (m <= static_cast<std::uint32_t>(kSwSM) && short_ok && short_rest == 0 &&
            s_nd <= static_cast<std::uint32_t>(kSwThreads))
        {
            if (!ready)
            {
                clean = false;
                for (int k = tid; k < kSwSH; k += kSwThreads)
                {
                    sh.t.cell[k] = kWinNone;
                    sh.t.key[k] = ~0ull;
                }
                if (tid == 0)
                {
                    sh.t.ne[0] = sh.t.ne[1] = m;
                    sh.t.out[0] = sh.t.out[1] = sh.t.nu[0] = sh.t.nu[1] = 0;
                    sh.t.over = 0;
                }
                __syncthreads();
            }
            ready = sw_short(G, B, sh, lst, near, open_rec, S, wst, m, q, Vmax, s_T, s_p, s_nd, dc, dk, dc2, dk2, lvc,
                             lvk, s_nl, level_of, out_F, s_V, s_m);
            q ^= 1u;
            if (ready)
            {
                short_back = 0;
                std::uint32_t* t1 = dc;
                dc = dc2;
                dc2 = t1;
                float* t2 = dk;
                dk = dk2;
                dk2 = t2;
                continue;
            }
            // given up (a second round, or too many cells): soon tried again,
            // later where it keeps giving up
            short_back = min(short_back + 1, 4);
            short_rest = (1 << short_back) - 1;
        }
        else if (short_rest > 0)
            --short_rest;
        ready = near.ok = false;
        __syncthreads();
        const bool narrow = m <= s_mlim;
        if (tid == 0)
        {
            for (int k = 0; k < 12; ++k) sh.cnt[k] = 0;
            s_nar = SwNarrowCtl{m, 0, 0, 0, 0, 0, {0, 0}, {0, 0}};
        }
        if (narrow && tid < 32)
        {
            // running maximum up to every FIFO entry
            float run = -INFINITY;
            for (std::uint32_t g0 = 0; g0 < m; g0 += 32)
            {
                const std::uint32_t g = g0 + tid;
                float v = g < m ? sh.fv[g] : -INFINITY;
                for (int o = 1; o < 32; o <<= 1)
                {
                    const float y = __shfl_up_sync(0xffffffffu, v, o);
                    if (tid >= o) v = fmaxf(v, y);
                }
                v = fmaxf(v, run);
                if (g < m) sh.n.pm[g] = v;
                run = __shfl_sync(0xffffffffu, v, 31);
            }
        }
        __syncthreads();
        const std::uint32_t sweep = s_sweep;
        if (narrow)
        {
            if (!clean)
            {
                sw_narrow_clear(sh.n);
                __syncthreads();
            }
            clean = sw_narrow(G, B, sh, s_nar, lst, open_rec, S, wst, m, Vmax, s_T, s_p, s_nd, dc, dk, dc2, dk2, lvc, lvk,
                              s_nl, level_of, out_F, s_V, s_m, s_mlim);
            if (clean)
            {
                std::uint32_t* t1 = dc;
                dc = dc2;
                dc2 = t1;
                float* t2 = dk;
                dk = dk2;
                dk2 = t2;
                continue;
            }
            __syncthreads();
            if (tid == 0) s_mlim = max(64u, m / 2);
        }
        else if (tid == 0) s_mlim = min(static_cast<std::uint32_t>(kSwNM), s_mlim + s_mlim / 16 + 1);
        clean = false;
        if (tid == 0)
            for (int k = 0; k < 12; ++k) sh.cnt[k] = 0;
        // the next greater FIFO value after each index (1-based, m + 1:
        // none): every thread looks up to 32 entries ahead; one thread
        // finishes the rest right to left with pointer jumps (entries
        // g + 1 .. g + 32 are known not greater)
        if (m > kSwScan)
        {
            for (std::uint32_t g = 1 + tid; g <= m; g += kSwThreads)
            {
                const float v = sh.fv[g - 1];
                const std::uint32_t lim = min(m + 1, g + 33);
                std::uint32_t n = g + 1;
                while (n < lim && !(sh.fv[n - 1] > v)) ++n;
                sh.w.ng[g] = static_cast<std::uint16_t>((n < lim || lim == m + 1) ? n : 0u);
            }
            __syncthreads();
            if (tid == 0)
            {
                sh.w.ng[m + 1] = static_cast<std::uint16_t>(m + 1);
                for (std::uint32_t g = m; g >= 1; --g)
                    if (sh.w.ng[g] == 0)
                    {
                        std::uint32_t n = g + 33;
                        while (n <= m && !(sh.fv[n - 1] > sh.fv[g - 1])) n = sh.w.ng[n];
                        sh.w.ng[g] = static_cast<std::uint16_t>(n);
                    }
            }
        }
        __syncthreads();
        auto push_list = [&](std::uint32_t* list, int which, std::uint32_t c) {
            const std::uint32_t k = atomicAdd(&sh.cnt[which], 1u);
            if (k < static_cast<std::uint32_t>(kSwL)) list[k] = c;
            else sh.cnt[5] = 1;
        };
        // the same for a whole warp at once (lanes with `want`): one atomic
        auto push_warp = [&](std::uint32_t* list, int which, bool want, std::uint32_t c) {
            const unsigned b = __ballot_sync(0xffffffffu, want);
            if (!b) return;
            const int lane = tid & 31;
            const int lead = __ffs(b) - 1;
            std::uint32_t base = 0;
            if (lane == lead) base = atomicAdd(&sh.cnt[which], static_cast<std::uint32_t>(__popc(b)));
            base = __shfl_sync(0xffffffffu, base, lead);
            if (want)
            {
                const std::uint32_t k = base + __popc(b & ((1u << lane) - 1u));
                if (k < static_cast<std::uint32_t>(kSwL)) list[k] = c;
                else sh.cnt[5] = 1;
            }
        };
        // FIFO entries: pops (g, 1)
        for (std::uint32_t g0 = 0; g0 < m; g0 += kSwThreads)
        {
            const std::uint32_t g = g0 + tid;
            std::uint32_t c = 0;
            if (g < m)
            {
                c = sh.fc[g];
                B.ev[c] = SwEv{sw_hi(g + 1, 1, 0.0f), sweep, sh.fv[g]};
            }
            push_warp(sh.w.la, 0, g < m, c);
        }
        // heap cells discovered earlier: those below Vmax pop in this sweep
        {
            const std::uint32_t nd = s_nd;
            constexpr int kU = 4;
            for (std::uint32_t t0 = 0; t0 < nd; t0 += kSwThreads * kU)
            {
                std::uint32_t cs[kU];
                float ks[kU];
#pragma unroll
                for (int u = 0; u < kU; ++u)
                {
                    const std::uint32_t t = t0 + u * kSwThreads + tid;
                    cs[u] = t < nd ? dc[t] : 0u;
                    ks[u] = t < nd ? dk[t] : INFINITY;
                }
#pragma unroll
                for (int u = 0; u < kU; ++u)
                {
                    const bool in = t0 + u * kSwThreads + tid < nd;
                    const bool pops = in && ks[u] < Vmax;
                    if (pops)
                    {
                        B.ev[cs[u]] = SwEv{sw_hi(sw_ng(sh, m, 1, ks[u]), 0, ks[u]), sweep, ks[u]};
                    }
                    push_warp(sh.w.la, 0, pops, cs[u]);
                    // survivors: compacted with one atomic per warp
                    const bool keep = in && !pops;
                    const unsigned b = __ballot_sync(0xffffffffu, keep);
                    if (b)
                    {
                        const int lane = tid & 31, lead = __ffs(b) - 1;
                        std::uint32_t base = 0;
                        if (lane == lead) base = atomicAdd(&sh.cnt[3], static_cast<std::uint32_t>(__popc(b)));
                        base = __shfl_sync(0xffffffffu, base, lead);
                        if (keep)
                        {
                            const std::uint32_t k2 = base + __popc(b & ((1u << lane) - 1u));
                            dc2[k2] = cs[u];
                            dk2[k2] = ks[u];
                        }
                    }
                }
            }
        }
        // list cells below Vmax (the sorted list from s_p on) pop too
        for (;;)
        {
            const std::int64_t p0 = s_p;
            const std::int64_t q = p0 + tid;
            bool past = q >= G.nsorted;
            bool pops = false;
            std::uint32_t c = 0;
            if (!past)
            {
                const float4 o = G.ordRec[q];
                if (!(o.x < Vmax)) past = true;
                else if (o.y < S)
                {
                    c = __float_as_uint(o.z);
                    B.ev[c] = SwEv{sw_hi(sw_ng(sh, m, 1, o.x), 0, o.x), sweep, o.x};
                    pops = true;
                }
            }
            push_warp(sh.w.la, 0, pops, c);
            if (tid == 0) sh.red_p = G.nsorted + 1;
            __syncthreads();
            if (past) atomicMin(reinterpret_cast<unsigned long long*>(&sh.red_p), static_cast<unsigned long long>(q));
            __syncthreads();
            const std::int64_t stop = sh.red_p;
            __syncthreads();
            if (stop <= G.nsorted)
            {
                if (tid == 0) s_p = stop;
                break;
            }
            if (tid == 0) s_p = p0 + kSwThreads;
            __syncthreads();
        }
        __syncthreads();
        // rounds: re-evaluate the not-yet-queued cells next to changed pops
        std::uint32_t* la = sh.w.la;
        std::uint32_t* lb = sh.w.lb;
        int rounds = 0;
        for (;;)
        {
            // (every thread has read the flag before a list of this round can
            // overflow and set it)
            const std::uint32_t nch = min(sh.cnt[0], static_cast<std::uint32_t>(kSwL));
            if (__syncthreads_or(nch == 0 || sh.cnt[5])) break;
            // a sweep settles in two or three rounds; one that has not after
            // 64 leaves the window to the sequential rules
            if (++rounds > 64)
            {
                __syncthreads();
                if (tid == 0) sh.cnt[5] = 1;
                __syncthreads();
                break;
            }
            const std::uint32_t round = sweep + static_cast<std::uint32_t>(rounds);
            for (std::uint32_t t = tid; t < nch * 8; t += kSwThreads)
            {
                const std::uint32_t c = la[t >> 3];
                const int dd = static_cast<int>(t & 7);
                const int r0 = static_cast<int>(c / static_cast<std::uint32_t>(G.nc));
                const int c0 = static_cast<int>(c - static_cast<std::uint32_t>(r0) * G.nc);
                int rr, cc;
                if (!fill_nb(G.nr, G.nc, G.per_ns, G.per_ew, r0, c0, dd, rr, cc)) continue;
                const std::uint32_t j = static_cast<std::uint32_t>(rr) * G.nc + cc;
                // every load the evaluation needs, issued before any is used:
                // j's record and state, the records of its eight neighbours
                std::uint32_t nbs[8];
#pragma unroll
                for (int d = 0; d < 8; ++d)
                {
                    int r2, c2;
                    nbs[d] = fill_nb(G.nr, G.nc, G.per_ns, G.per_ew, rr, cc, d, r2, c2)
                                 ? static_cast<std::uint32_t>(r2) * G.nc + c2
                                 : kWinNone;
                }
                const float4 qj = sw_record(G.rec + j);
                SwEv evs[8];
#pragma unroll
                for (int d = 0; d < 8; ++d) evs[d] = B.ev[nbs[d] != kWinNone ? nbs[d] : j];
                const SwEv self = B.ev[j];
                const float zj = qj.x;
                if (!open_rec(qj)) continue;
                // one thread per cell and round: the cell's records have a
                // single writer within the round (an older mark: first
                // visit in this sweep, listed for the finalisation)
                const std::uint32_t prev_mark = atomicExch(&B.mk_c[j], round);
                if (prev_mark == round) continue;
                if (prev_mark <= sweep) push_list(sh.w.lt, 2, j);
                // the neighbour of j that pops first, and its direction to j
                std::uint64_t bh = ~0ull;
                std::uint32_t bl = ~0u;
                float bval = 0.0f;
                int bk = 8;
#pragma unroll
                for (int d = 0; d < 8; ++d)
                {
                    if (nbs[d] == kWinNone || evs[d].st != sweep) continue;
                    const std::uint64_t h = evs[d].hi;
                    const std::uint32_t l = ((h >> 32) & 1u) ? 0u : nbs[d];
                    const int k = (d + 4) & 7;
                    if (h < bh || (h == bh && (l < bl || (l == bl && k < bk))))
                    {
                        bh = h;
                        bl = l;
                        bk = k;
                        bval = evs[d].val;
                    }
                }
                const bool was_ev = self.st == sweep;
                if (bk == 8)
                {
                    // no pop next to it any more: not discovered in this sweep
                    B.te_st[j] = 0;
                    if (was_ev)
                    {
                        B.ev[j].st = 0;
                        push_list(lb, 1, j);
                    }
                    continue;
                }
                B.te[j] = SwTe{bh, bl, bval};
                B.te_k[j] = static_cast<std::uint8_t>(bk);
                B.te_st[j] = sweep;
                bool ev = false;
                std::uint64_t nh = 0;
                if (!(zj <= bval))
                {
                    const std::uint32_t gd = static_cast<std::uint32_t>(bh >> 33);
                    const std::uint32_t gpush = ((bh >> 32) & 1u) ? gd + 1 : gd;
                    const std::uint32_t g = sw_ng(sh, m, gpush, zj);
                    if (g <= m)
                    {
                        ev = true;
                        nh = sw_hi(g, 0, zj);
                    }
                }
                if (ev)
                {
                    if (!was_ev || self.hi != nh)
                    {
                        B.ev[j] = SwEv{nh, sweep, zj};
                        push_list(lb, 1, j);
                    }
                }
                else if (was_ev)
                {
                    B.ev[j].st = 0;
                    push_list(lb, 1, j);
                }
            }
            __syncthreads();
            if (tid == 0)
            {
                sh.cnt[0] = sh.cnt[1];
                sh.cnt[1] = 0;
            }
            std::uint32_t* t = la;
            la = lb;
            lb = t;
            __syncthreads();
        }
        __syncthreads();
        if (sh.cnt[5] || sh.cnt[2] > static_cast<std::uint32_t>(kSwL))
        {
            if (tid == 0) s_status = kWinOverflow;
            __syncthreads();
            break;
        }
        // finalize: pops, next FIFO, heap cells
        float vmax_pop = -INFINITY;
        for (std::uint32_t g = tid; g < m; g += kSwThreads)
        {
            const std::uint32_t c = sh.fc[g];
            out_F[c] = sh.fv[g];
            vmax_pop = fmaxf(vmax_pop, sh.fv[g]);
        }
        const std::uint32_t nt = sh.cnt[2];
        for (std::uint32_t t = tid; t < nt; t += kSwThreads)
        {
            const std::uint32_t j = sh.w.lt[t];
            const std::uint32_t tst = B.te_st[j];
            const float zj = G.rec[j].x;
            const SwEv e = B.ev[j];
            const SwTe d = B.te[j];
            const int dk_dir = B.te_k[j];
            if (tst != sweep) continue;
            if (e.st == sweep)
            {
                set_queued(j);
                vmax_pop = fmaxf(vmax_pop, zj);
            }
            else if (zj <= d.val)
            {
                const std::uint32_t s2 = atomicAdd(&sh.cnt[4], 1u);
                if (s2 < static_cast<std::uint32_t>(kSwFQ))
                {
                    const int k = dk_dir;
                    sh.w.nc[s2] = j;
                    sh.w.nv[s2] = raise_from(d.val, G.eps, (k & 1) ? G.Ld : G.L);
                    sh.w.nhi[s2] = d.hi;
                    sh.w.nlo[s2] = d.lo;
                    sh.w.nk[s2] = static_cast<std::uint8_t>(k);
                }
                set_queued(j);
            }
            else
            {
                if (zj < s_T)
                {
                    const std::uint32_t s2 = atomicAdd(&sh.cnt[3], 1u);
                    dc2[s2] = j;
                    dk2[s2] = zj;
                }
                else
                {
                    const int k = level_of(zj);
                    const std::uint32_t s2 = s_nl[k] + atomicAdd(&sh.cnt[7 + k], 1u);
                    lvc(k)[s2] = j;
                    lvk(k)[s2] = zj;
                }
                set_queued(j);
            }
        }
        // the largest value popped: the FIFO's (list and earlier heap pops
        // are below Vmax, the FIFO's largest) or a discovered cell's
        for (int o = 16; o > 0; o >>= 1) vmax_pop = fmaxf(vmax_pop, __shfl_down_sync(0xffffffffu, vmax_pop, o));
        if ((tid & 31) == 0) sh.red_v[tid >> 5] = vmax_pop;
        __syncthreads();
        const std::uint32_t mn = sh.cnt[4];
        if (tid == 0)
        {
            float v = s_V;
            for (int k = 0; k < kSwThreads / 32; ++k) v = fmaxf(v, sh.red_v[k]);
            s_V = v;
            s_nd = sh.cnt[3];
            for (int k = 0; k < kSwLv; ++k) s_nl[k] += sh.cnt[7 + k];
            if (mn > static_cast<std::uint32_t>(kSwFQ)) s_status = kWinOverflow;
        }
        __syncthreads();
        if (s_status != kWinOk) break;
        // the next FIFO in push order (discoverer's T, direction): each entry
        // counts the entries before it (keys are distinct); up to 32 entries
        // within warp 0 by shuffles, past 64 by a bitonic sort of indices
        // (ng is free until the next sweep builds it)
        if (mn > 64)
        {
            const std::uint32_t P = 1u << (32 - __clz(mn - 1));
            for (std::uint32_t t = tid; t < P; t += kSwThreads) sh.w.ng[t] = static_cast<std::uint16_t>(t);
            __syncthreads();
            // a after b in push order (indices past mn last)
            auto after = [&](std::uint32_t a, std::uint32_t b) {
                if (a >= mn) return b < mn || a > b;
                if (b >= mn) return false;
                const std::uint64_t ah = sh.w.nhi[a], bh = sh.w.nhi[b];
                if (ah != bh) return ah > bh;
                const std::uint32_t al = sh.w.nlo[a], bl = sh.w.nlo[b];
                if (al != bl) return al > bl;
                return sh.w.nk[a] > sh.w.nk[b];
            };
            for (std::uint32_t k = 2; k <= P; k <<= 1)
                for (std::uint32_t j = k >> 1; j > 0; j >>= 1)
                {
                    for (std::uint32_t i = tid; i < P; i += kSwThreads)
                    {
                        const std::uint32_t l = i ^ j;
                        if (l > i)
                        {
                            const std::uint32_t a = sh.w.ng[i], b = sh.w.ng[l];
                            if (after(a, b) == ((i & k) == 0))
                            {
                                sh.w.ng[i] = static_cast<std::uint16_t>(b);
                                sh.w.ng[l] = static_cast<std::uint16_t>(a);
                            }
                        }
                    }
                    __syncthreads();
                }
            for (std::uint32_t r = tid; r < mn; r += kSwThreads)
            {
                const std::uint32_t a = sh.w.ng[r];
                sh.fc[r] = sh.w.nc[a];
                sh.fv[r] = sh.w.nv[a];
            }
        }
        else if (mn <= 32)
        {
            if (tid < 32)
            {
                const bool in = static_cast<std::uint32_t>(tid) < mn;
                const std::uint64_t ah = in ? sh.w.nhi[tid] : ~0ull;
                const std::uint32_t al = in ? sh.w.nlo[tid] : ~0u;
                const std::uint32_t ak = in ? sh.w.nk[tid] : 255u;
                const std::uint32_t ac = in ? sh.w.nc[tid] : 0u;
                const float av = in ? sh.w.nv[tid] : 0.0f;
                std::uint32_t rank = 0;
                for (int b = 0; b < 32; ++b)
                {
                    const std::uint64_t bh = __shfl_sync(0xffffffffu, ah, b);
                    const std::uint32_t bl = __shfl_sync(0xffffffffu, al, b);
                    const std::uint32_t bk = __shfl_sync(0xffffffffu, ak, b);
                    if (static_cast<std::uint32_t>(b) < mn &&
                        (bh < ah || (bh == ah && (bl < al || (bl == al && bk < ak)))))
                        ++rank;
                }
                if (in)
                {
                    sh.fc[rank] = ac;
                    sh.fv[rank] = av;
                }
            }
        }
        else
        for (std::uint32_t a = tid; a < mn; a += kSwThreads)
        {
            const std::uint64_t ah = sh.w.nhi[a];
            const std::uint32_t al = sh.w.nlo[a];
            const std::uint8_t ak = sh.w.nk[a];
            std::uint32_t rank = 0;
            for (std::uint32_t b = 0; b < mn; ++b)
            {
                const std::uint64_t bh = sh.w.nhi[b];
                if (bh < ah || (bh == ah && (sh.w.nlo[b] < al || (sh.w.nlo[b] == al && sh.w.nk[b] < ak)))) ++rank;
            }
            sh.fc[rank] = sh.w.nc[a];
            sh.fv[rank] = sh.w.nv[a];
        }
        __syncthreads();
        if (tid == 0) s_m = mn;
        {
            std::uint32_t* t1 = dc;
            dc = dc2;
            dc2 = t1;
            float* t2 = dk;
            dk = dk2;
            dk2 = t2;
        }
        __syncthreads();
    }
    if (tid == 0) *ctr = s_ctr;
    __syncthreads();
    *next = s_next;  // every thread: the caller's control flow stays uniform
    const int status = static_cast<int>(s_status);
    __syncthreads();  // s_* are reused by the next call
    return status;
}

}  // namespace
}  // namespace lsdtt_gb300
