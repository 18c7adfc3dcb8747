// stack.cu -- s-vector, contributing-cell counts, depths, heights and the
// Kahn topological order of the D8 receiver forest, all without a
// level-by-level sweep.
//
// 1. Euler tour. The reference's s-vector (src/cpu/lsdtt_flowinfo_cpu.cpp:
//    1544-1731) is a DFS preorder from each outlet in row-major order with
//    donors visited in ascending flat index. That preorder is the order of
//    "enter" events on the Euler tour of the forest whose children lists are
//    sorted ascending and whose trees are chained in outlet order. Each valid
//    cell c owns two tour nodes, enter(c) = 2c and exit(c) = 2c+1, and the
//    successor of every node follows from first child / next sibling /
//    parent / next outlet.
// 2. List ranking by a sparse ruling set: about one node in 32 (and the head)
//    starts a walk to the next ruler, the rulers' list is ranked
//    recursively, then every node adds its ruler's rank. With weights
//    (enter: +1, exit: 0) the prefix is the preorder index; with (+1, -1)
//    it is the depth. s_vector_start = prefix at enter, s_vector_size =
//    prefix at exit - prefix at enter, depth = signed prefix at enter.
// 3. Kahn order (build_topological_order, :1428-1522). The FIFO processes
//    level L_k (cells whose longest path from a headwater is k) before
//    L_{k+1}, and L_{k+1} is the list of receivers pushed by L_k in L_k
//    order, each pushed by its last-processed donor. By induction the order
//    inside every level is the order of the flat index of a single
//    headwater per cell: the deepest headwater of its subtree, the largest
//    flat index among equally deep ones. Both the height and that headwater
//    are one range-max over the cell's s-vector interval of the key
//    (depth << 32 | flat). The order is then a stable radix sort by
//    (height, headwater).

#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "engine.cuh"

namespace lsdtt_gb300
{
namespace
{

constexpr std::uint32_t kEnd = 0xffffffffu;
constexpr std::uint32_t kNone = 0xffffffffu;
constexpr unsigned kErrCycle = 5;
// Mean sublist length of the ruling set (a power of two). The first level's
// walk is bound by its longest sublist, ~kRuler ln(#rulers) dependent steps;
// a smaller kRuler shortens it but adds rulers and levels. Of 16, 32 and 64,
// 32 gave the fastest s-vector on an 89.5 M-cell ensemble. The ruler
// buffers take 24 B per ruler, sized for four times the mean count.
constexpr int kRuler = 32;
constexpr int kSerialLimit = 96;  // rank lists this short with one thread

__device__ __forceinline__ bool is_ruler(std::uint32_t v)
{
    // Spread rulers pseudo-randomly so sublists stay short on any layout.
    std::uint32_t h = v * 0x9E3779B1u;
    h ^= h >> 15;
    return (h & (kRuler - 1)) == 0;
}

// Sorted donor list of a valid cell: ascending flat index, de-duplicated
// (a donor matches exactly one direction, see donors_kernel).
__device__ int donor_list(const Grid& g, const std::uint8_t* __restrict__ mask, const std::uint8_t* __restrict__ dir,
                          std::int64_t flat, std::int64_t out[8])
{
    const int row = static_cast<int>(flat / g.nc), col = static_cast<int>(flat % g.nc);
    int k = 0;
    if (is_interior(g, row, col))
    {
        // NW, N, NE, W, E, SW, S, SE: ascending flat order; code of each and
        // the code that points back (opposite).
        const int order[8] = {7, 0, 1, 6, 2, 5, 4, 3};
#pragma unroll
        for (int i = 0; i < 8; ++i)
        {
            const int d = order[i];
            const std::int64_t nf = flat + static_cast<std::int64_t>(d8_dr(d)) * g.nc + d8_dc(d);
            if (dir[nf] == ((d + 4) & 7)) out[k++] = nf;  // a masked cell has no direction
        }
        return k;
    }
    for (int d = 0; d < 8; ++d)
    {
        const Step s = resolve_step(g, row, col, d);
        if (s.kind != 1) continue;
        const std::int64_t nf = static_cast<std::int64_t>(s.r) * g.nc + s.c;
        if (nf == flat || !mask[nf] || dir[nf] != ((d + 4) & 7)) continue;
        bool dup = false;
        for (int i = 0; i < k; ++i) dup |= (out[i] == nf);
        if (!dup) out[k++] = nf;
    }
    for (int i = 1; i < k; ++i)
    {
        const std::int64_t key = out[i];
        int j = i;
        while (j > 0 && out[j - 1] > key) { out[j] = out[j - 1]; --j; }
        out[j] = key;
    }
    return k;
}

// first child / next sibling links of the cell at `flat` (an index into the
// grid g's planes; written links get `base` added). next_sibling of each
// donor is written by its (unique) receiver. Interior cells scan their eight
// neighbours in ascending flat order (NW, N, NE, W, E, SW, S, SE) and chain
// the donors as they are found; edge cells take donor_list.
__device__ __forceinline__ void link_cell(const Grid& g, const std::uint8_t* __restrict__ mask,
                                          const std::uint8_t* __restrict__ dir, std::int64_t flat, std::int64_t base,
                                          std::uint32_t* __restrict__ first_child,
                                          std::uint32_t* __restrict__ next_sib)
{
    const int row = static_cast<int>(flat / g.nc), col = static_cast<int>(flat % g.nc);
    std::uint32_t first = kNone, prev = kNone;
    auto chain = [&](std::int64_t nf) {
        const std::uint32_t v = static_cast<std::uint32_t>(base + nf);
        if (prev == kNone) first = v;
        else next_sib[prev] = v;
        prev = v;
    };
    if (is_interior(g, row, col))
    {
        const int order[8] = {7, 0, 1, 6, 2, 5, 4, 3};  // the codes of NW, N, NE, W, E, SW, S, SE
#pragma unroll
        for (int i = 0; i < 8; ++i)
        {
            const int d = order[i];
            const std::int64_t nf = flat + static_cast<std::int64_t>(d8_dr(d)) * g.nc + d8_dc(d);
            if (dir[nf] == ((d + 4) & 7)) chain(nf);  // a masked cell has no direction
        }
    }
    else
    {
        std::int64_t d[8];
        const int k = donor_list(g, mask, dir, flat, d);
        for (int i = 0; i < k; ++i) chain(d[i]);
    }
    first_child[base + flat] = first;
    if (prev != kNone) next_sib[prev] = kNone;
}

__global__ void links_kernel(Grid g, const std::uint8_t* __restrict__ mask, const std::uint8_t* __restrict__ dir,
                             std::uint32_t* __restrict__ first_child, std::uint32_t* __restrict__ next_sib)
{
    LSDTT_COUNT();
    const std::int64_t flat = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (flat >= g.n || !mask[flat]) return;
    link_cell(g, mask, dir, flat, 0, first_child, next_sib);
}

// links_kernel for a packed ensemble: each member's donors in its own
// geometry, written as packed indices. Blocks are kPackAlign cells, so each
// lies in one member.
__global__ void links_packed(Packed P, const std::uint8_t* __restrict__ mask, const std::uint8_t* __restrict__ dir,
                             std::uint32_t* __restrict__ first_child, std::uint32_t* __restrict__ next_sib)
{
    LSDTT_COUNT();
    const std::int64_t flat = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (flat >= P.n || !mask[flat]) return;
    const PackedMember& M = P.m[P.blk_member[blockIdx.x]];
    const std::int64_t local = flat - M.base;
    if (local >= static_cast<std::int64_t>(M.nr) * M.nc) return;
    link_cell(member_grid(M), mask + M.base, dir + M.base, local, M.base, first_child, next_sib);
}

__global__ void root_links_kernel(const std::int64_t* __restrict__ outlets, const std::int64_t* __restrict__ n_out,
                                  std::uint32_t* __restrict__ next_sib, std::uint32_t* __restrict__ head)
{
    LSDTT_COUNT();
    const std::int64_t n = *n_out;
    const std::int64_t t0 = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t0 == 0) *head = n > 0 ? static_cast<std::uint32_t>(2 * outlets[0]) : kEnd;
    // (strided: the count is on the device, far below one thread a cell)
    for (std::int64_t i = t0; i < n; i += static_cast<std::int64_t>(gridDim.x) * blockDim.x)
        next_sib[outlets[i]] = (i + 1 < n) ? static_cast<std::uint32_t>(outlets[i + 1]) : kNone;
}

// Successor of every tour node. For a root the "next sibling" link holds the
// next outlet, and a root's exit with no next outlet ends the list.
__global__ void succ_kernel(Grid g, const std::uint8_t* __restrict__ mask, const std::int64_t* __restrict__ receiver,
                            const std::uint32_t* __restrict__ first_child, const std::uint32_t* __restrict__ next_sib,
                            std::uint32_t* __restrict__ succ)
{
    LSDTT_COUNT();
    const std::int64_t flat = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (flat >= g.n) return;
    if (!mask[flat])
    {
        succ[2 * flat] = kEnd;
        succ[2 * flat + 1] = kEnd;
        return;
    }
    const std::uint32_t fc = first_child[flat];
    const std::uint32_t ns = next_sib[flat];
    const std::int64_t p = receiver[flat];
    succ[2 * flat] = (fc != kNone) ? 2u * fc : static_cast<std::uint32_t>(2 * flat + 1);
    if (ns != kNone) succ[2 * flat + 1] = 2u * ns;
    else if (p >= 0) succ[2 * flat + 1] = static_cast<std::uint32_t>(2 * p + 1);
    else succ[2 * flat + 1] = kEnd;
}

struct RankLevel
{
    std::uint32_t n;                 // node capacity of this level
    const std::uint32_t* succ;       // [n]
    const std::int32_t* w0;          // [n] or null: parity weights
    const std::int32_t* w1;          // [n] or null
    const std::uint8_t* cell_mask;   // level 0: node v valid iff cell_mask[v>>1]
    const std::uint32_t* head;       // device scalar
    const std::uint32_t* count;      // device scalar: valid nodes at this level (null: n)
};

__device__ __forceinline__ void weights(const RankLevel& L, std::uint32_t v, int& a, int& b)
{
    if (L.w0) { a = L.w0[v]; b = L.w1[v]; }
    else { a = (v & 1u) ? 0 : 1; b = (v & 1u) ? -1 : 1; }
}

__device__ __forceinline__ bool node_valid(const RankLevel& L, std::uint32_t v)
{
    if (L.cell_mask) return L.cell_mask[v >> 1] != 0;
    return v < *L.count;
}

// Per node of a ranking level: the ruler whose walk reached it and the two
// prefixes from that ruler, one record (a walk step writes one sector, not
// three). On the tour itself the prefixes are the counts of enter and exit
// nodes passed, which fit half a word each: a walk that reaches kWalkMax nodes
// goes on as a ruler of its own.
struct alignas(16) RankRec
{
    std::uint32_t owner;
    std::int32_t loc0, loc1, pad;
    __device__ static RankRec make(std::uint32_t i, int a0, int a1) { return RankRec{i, a0, a1, 0}; }
};
struct alignas(8) TourRec
{
    std::uint32_t owner;
    std::uint32_t passed;  // enter nodes | exit nodes << 16
    // (a0: enter nodes; a1: enter - exit nodes)
    __device__ static TourRec make(std::uint32_t i, int a0, int a1)
    {
        return TourRec{i, static_cast<std::uint32_t>(a0) | static_cast<std::uint32_t>(a0 - a1) << 16};
    }
    __device__ int loc0() const { return static_cast<int>(passed & 0xffffu); }
    __device__ int loc1() const { return static_cast<int>(passed & 0xffffu) - static_cast<int>(passed >> 16); }
};
constexpr std::uint32_t kWalkMax = 255;  // nodes of a tour walk before it splits

// Ruler compaction in one pass: each thread takes 16 consecutive nodes, a
// block scans its rulers and claims a range of the ruler list with one
// atomic (ruler numbers then depend on block order; the ranks do not). Also
// counts the level's valid nodes (cnt[2]) for the coverage check.
constexpr int kCompactPer = 16;

template <class Rec>
__global__ void __launch_bounds__(256) ruler_compact(RankLevel L, std::uint32_t cap, std::uint32_t* __restrict__ rulers,
                                                     Rec* __restrict__ rec, std::uint32_t* __restrict__ cnt)
{
    LSDTT_COUNT();
    __shared__ unsigned wsum[8], wval[8], s_base;
    const std::uint32_t head = *L.head;
    const std::uint32_t v0 = (blockIdx.x * blockDim.x + threadIdx.x) * kCompactPer;
    unsigned rmask = 0, nvalid = 0;
#pragma unroll
    for (int j = 0; j < kCompactPer; ++j)
    {
        const std::uint32_t v = v0 + j;
        if (v < L.n && node_valid(L, v))
        {
            ++nvalid;
            if (is_ruler(v) || v == head) rmask |= 1u << j;
        }
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned nr = __popc(rmask);
    unsigned incl = nr;
    for (int o = 1; o < 32; o <<= 1)
    {
        const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    unsigned val = nvalid;
    for (int o = 16; o > 0; o >>= 1) val += __shfl_down_sync(0xffffffffu, val, o);
    if (lane == 31) wsum[w] = incl;
    if (lane == 0) wval[w] = val;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        unsigned tot = 0, tv = 0;
        for (int k = 0; k < static_cast<int>(blockDim.x >> 5); ++k)
        {
            const unsigned t = wsum[k];
            wsum[k] = tot;
            tot += t;
            tv += wval[k];
        }
        s_base = tot ? atomicAdd(&cnt[0], tot) : 0u;
        if (tv) atomicAdd(&cnt[2], tv);
    }
    __syncthreads();
    std::uint32_t pos = s_base + wsum[w] + incl - nr;
#pragma unroll
    for (int j = 0; j < kCompactPer; ++j)
        if ((rmask >> j) & 1u)
        {
            if (pos < cap)
            {
                rulers[pos] = v0 + j;
                rec[v0 + j].owner = pos;
            }
            ++pos;  // a count above cap is reported by ruler_checks
        }
}

// After the walks: too many rulers, or walks that did not cover every valid
// node of the level (a successor structure that is not one list).
// Adds the rulers that walks split off to the level's count.
__global__ void ruler_checks(std::uint32_t* cnt, std::uint32_t cap, unsigned long long* err)
{
    LSDTT_COUNT();
    cnt[0] += cnt[4];
    if (cnt[0] > cap) raise_error(err, 9, cnt[0]);
    else if (cnt[3] != cnt[2]) raise_error(err, kErrCycle, 2);
}

// A walk from ruler i to the next ruler. A node of the list is a ruler iff
// is_ruler(v) or it is the head (ruler_compact), so the stop test needs no
// load. The chain of successors bounds it, so a step loads the next node before
// it writes this one's record, and a tour walk is split outside the loop (33 M
// nodes 873 us with both inside, now 458; 16-byte records took 640). One ruler a
// thread, in the order of the rulers: the walks of a block then keep to the
// same lines (taking the next ruler as soon as a walk ends spread them, 5.8 ms
// against 4.0 on an ensemble's tour).
template <class Rec>
__global__ void __launch_bounds__(128) ruler_walk(RankLevel L, const std::uint32_t* __restrict__ rulers,
                                                  std::uint32_t* __restrict__ cnt, Rec* __restrict__ rec,
                                                  std::int32_t* __restrict__ sub0,
                                                  std::int32_t* __restrict__ sub1, std::uint32_t* __restrict__ nxt,
                                                  std::uint32_t* __restrict__ next_head, std::uint32_t cap,
                                                  unsigned long long* __restrict__ err)
{
    LSDTT_COUNT();
    constexpr bool kTour = sizeof(Rec) == sizeof(TourRec);
    std::uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const std::uint32_t nr = min(cnt[0], cap);
    if (i >= nr) return;
    const std::uint32_t head = *L.head;
    std::uint32_t v = rulers[i];
    if (v == head) *next_head = i;
    int a0 = 0, a1 = 0;
    std::uint32_t steps = 0, limit = kTour ? kWalkMax : ~0u;
    for (;;)
    {
        do
        {
            const std::uint32_t u = L.succ[v];
            rec[v] = Rec::make(i, a0, a1);
            int w0, w1;
            if (kTour) { w0 = 1 - static_cast<int>(v & 1u); w1 = 1 - 2 * static_cast<int>(v & 1u); }
            else weights(L, v, w0, w1);
            a0 += w0;
            a1 += w1;
            v = u;
            ++steps;
        } while (v != kEnd && !is_ruler(v) && v != head && steps <= L.n && steps != limit);
        if (v == kEnd || is_ruler(v) || v == head || steps > L.n) break;
        // the walk goes on as ruler j
        const std::uint32_t j = nr + atomicAdd(&cnt[4], 1u);
        if (j >= cap) break;  // reported by ruler_checks
        sub0[i] = a0;
        sub1[i] = a1;
        nxt[i] = j;
        i = j;
        a0 = a1 = 0;
        limit += kWalkMax;
    }
    if (steps > L.n) raise_error(err, kErrCycle, 0);
    sub0[i] = a0;
    sub1[i] = a1;
    nxt[i] = (v == kEnd) ? kEnd : rec[v].owner;
    // coverage: the walks visit every valid node exactly once (one atomic per
    // converged group of lanes)
    const unsigned grp = __activemask();
    const unsigned tot = __reduce_add_sync(grp, steps);
    if ((threadIdx.x & 31) == static_cast<unsigned>(__ffs(grp) - 1)) atomicAdd(&cnt[3], tot);
}

// A level of up to kBlockLimit nodes ranked by one block: pointer jumping over
// the nodes' successors and the sums (and node counts) from a node to the end
// of the list, in shared memory. The recursion's last levels were five
// launches each for a few hundred nodes: 52 k tour nodes 100 us after the first
// level's walk, now 12.
constexpr std::uint32_t kBlockLimit = 12288;
constexpr int kBlockPer = 12;  // nodes per thread
struct BlockNode
{
    std::uint32_t next;
    std::int32_t s0, s1;
    std::uint32_t count;
};

__global__ void __launch_bounds__(1024) block_rank(RankLevel L, std::int32_t* __restrict__ p0,
                                                   std::int32_t* __restrict__ p1, unsigned long long* __restrict__ err)
{
    LSDTT_COUNT();
    extern __shared__ BlockNode node[];
    const std::uint32_t n = min(*L.count, L.n), head = *L.head;
    for (std::uint32_t v = threadIdx.x; v < n; v += 1024)
    {
        const std::uint32_t u = L.succ[v];
        node[v] = BlockNode{u < n ? u : kEnd, L.w0[v], L.w1[v], 1u};
    }
    __syncthreads();
    BlockNode own[kBlockPer];
    for (int round = 0; round < 15; ++round)
    {
        bool more = false;
#pragma unroll
        for (int k = 0; k < kBlockPer; ++k)
        {
            const std::uint32_t v = k * 1024u + threadIdx.x;
            if (k * 1024u >= n) break;  // (block-uniform)
            if (v >= n) continue;
            own[k] = node[v];
            if (own[k].next != kEnd)
            {
                const BlockNode b = node[own[k].next];
                own[k].next = b.next;
                own[k].s0 += b.s0;
                own[k].s1 += b.s1;
                own[k].count += b.count;
                more = true;
            }
        }
        if (!__syncthreads_or(more)) break;
#pragma unroll
        for (int k = 0; k < kBlockPer; ++k)
        {
            const std::uint32_t v = k * 1024u + threadIdx.x;
            if (k * 1024u >= n) break;
            if (v < n) node[v] = own[k];
        }
        __syncthreads();
    }
    if (n == 0) return;
    // One list from the head through every node, or the successors are not a
    // list (a cycle never ends, a part beside it is not counted).
    if (head >= n || node[head].next != kEnd || node[head].count != n)
    {
        if (threadIdx.x == 0) raise_error(err, kErrCycle, 2);
        for (std::uint32_t v = threadIdx.x; v < n; v += 1024) p0[v] = p1[v] = 0;
        return;
    }
    const std::int32_t t0 = node[head].s0, t1 = node[head].s1;
    for (std::uint32_t v = threadIdx.x; v < n; v += 1024)
    {
        p0[v] = t0 - node[v].s0;
        p1[v] = t1 - node[v].s1;
    }
}

__global__ void serial_rank(RankLevel L, std::int32_t* __restrict__ p0, std::int32_t* __restrict__ p1,
                            unsigned long long* __restrict__ err)
{
    LSDTT_COUNT();
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    std::uint32_t v = *L.head;
    int a0 = 0, a1 = 0;
    std::uint32_t steps = 0;
    while (v != kEnd && steps <= L.n)
    {
        p0[v] = a0;
        p1[v] = a1;
        int w0, w1;
        weights(L, v, w0, w1);
        a0 += w0;
        a1 += w1;
        v = L.succ[v];
        ++steps;
    }
    if (steps > L.n) raise_error(err, kErrCycle, 1);
}

__global__ void rank_finish(RankLevel L, const RankRec* __restrict__ rec, const std::int32_t* __restrict__ P0,
                            const std::int32_t* __restrict__ P1, std::uint32_t cap, std::int32_t* __restrict__ p0,
                            std::int32_t* __restrict__ p1, unsigned long long* __restrict__ err)
{
    LSDTT_COUNT();
    const std::uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= L.n || !node_valid(L, v)) return;
    const RankRec r = rec[v];
    const std::uint32_t o = r.owner;
    if (o >= cap)
    {
        // Not reached by any walk: the tour does not cover every valid node.
        raise_error(err, kErrCycle, 2);
        p0[v] = -1;
        p1[v] = 0;
        return;
    }
    p0[v] = P0[o] + r.loc0;
    p1[v] = P1[o] + r.loc1;
}

// Per-cell s-vector outputs, written straight from the level-0 ranking
// (sv_finish) or from its prefix arrays (sv_outputs). start and svec may be
// null (a caller that needs the counts and depths only).
struct SvOut
{
    Grid g;
    const std::uint8_t* mask;
    std::int64_t n_valid;
    std::int64_t* start;
    std::uint64_t* size;
    std::int32_t* depth;
    std::int64_t* svec;
};

__device__ __forceinline__ void sv_store(const SvOut& o, std::int64_t c, std::int32_t s, std::int32_t e,
                                         std::int32_t dep, unsigned long long* __restrict__ err)
{
    if (s < 0 || e <= s || static_cast<std::int64_t>(e) > o.n_valid)
    {
        raise_error(err, kErrCycle, 3);
        if (o.start) o.start[c] = kNodataReceiver;
        o.size[c] = 0;
        o.depth[c] = 0;
        return;
    }
    if (o.start) o.start[c] = s;
    o.size[c] = static_cast<std::uint64_t>(e - s);
    o.depth[c] = dep;
    if (o.svec) o.svec[s] = c;
}

__device__ __forceinline__ bool sv_masked(const SvOut& o, std::int64_t c)
{
    if (o.mask[c]) return false;
    if (o.start) o.start[c] = kNodataReceiver;
    o.size[c] = 0;
    o.depth[c] = -1;
    return true;
}

// rank_finish and sv_outputs in one pass over the cells of the level-0
// (Euler tour) list: cell c's enter and exit records are adjacent.
__global__ void sv_finish(RankLevel L, const TourRec* __restrict__ rec, const std::int32_t* __restrict__ P0,
                          const std::int32_t* __restrict__ P1, std::uint32_t cap, SvOut o,
                          unsigned long long* __restrict__ err)
{
    LSDTT_COUNT();
    const std::int64_t c = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= o.g.n || sv_masked(o, c)) return;
    const uint4 q = reinterpret_cast<const uint4*>(rec)[c];
    const TourRec a{q.x, q.y}, b{q.z, q.w};
    if (a.owner >= cap || b.owner >= cap)
    {
        // Not reached by any walk: the tour does not cover every valid node.
        raise_error(err, kErrCycle, 2);
        sv_store(o, c, -1, -1, 0, err);
        return;
    }
    sv_store(o, c, P0[a.owner] + a.loc0(), P0[b.owner] + b.loc0(), P1[a.owner] + a.loc1(), err);
}

// Recursive list ranking. p0/p1 receive the exclusive prefix sums of the two
// weights along the list starting at *L.head; with sv (the level-0 Euler
// tour of a grid, longer than kSerialLimit) the per-cell s-vector outputs are
// written instead and p0/p1 are not used.
template <class Rec>
cudaError_t rank_rulers(const RankLevel& L, std::int32_t* p0, std::int32_t* p1, Scratch& ws, unsigned long long* err,
                        cudaStream_t st, const SvOut* sv);

cudaError_t rank_list(const RankLevel& L, std::int32_t* p0, std::int32_t* p1, Scratch& ws,
                      unsigned long long* err, cudaStream_t st, const SvOut* sv = nullptr)
{
    if (sv) return rank_rulers<TourRec>(L, p0, p1, ws, err, st, sv);
    if (L.n <= static_cast<std::uint32_t>(kSerialLimit))
    {
        serial_rank<<<1, 32, 0, st>>>(L, p0, p1, err);
        return cudaGetLastError();
    }
    if (L.n <= kBlockLimit && L.count)
    {
        const int bytes = static_cast<int>(sizeof(BlockNode) * L.n);
        const cudaError_t e = cudaFuncSetAttribute(block_rank, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   static_cast<int>(sizeof(BlockNode) * kBlockLimit));
        if (e != cudaSuccess) return e;
        block_rank<<<1, 1024, bytes, st>>>(L, p0, p1, err);
        return cudaGetLastError();
    }
    return rank_rulers<RankRec>(L, p0, p1, ws, err, st, nullptr);
}

void launch_finish(const RankLevel& L, const TourRec* rec, const std::int32_t* P0, const std::int32_t* P1,
                   std::uint32_t cap, std::int32_t*, std::int32_t*, unsigned long long* err, cudaStream_t st,
                   const SvOut* sv)
{
    sv_finish<<<grid_blocks(sv->g.n, 256), 256, 0, st>>>(L, rec, P0, P1, cap, *sv, err);
}

void launch_finish(const RankLevel& L, const RankRec* rec, const std::int32_t* P0, const std::int32_t* P1,
                   std::uint32_t cap, std::int32_t* p0, std::int32_t* p1, unsigned long long* err, cudaStream_t st,
                   const SvOut*)
{
    rank_finish<<<grid_blocks(L.n, 256), 256, 0, st>>>(L, rec, P0, P1, cap, p0, p1, err);
}

template <class Rec>
cudaError_t rank_rulers(const RankLevel& L, std::int32_t* p0, std::int32_t* p1, Scratch& ws, unsigned long long* err,
                        cudaStream_t st, const SvOut* sv)
{
    const std::size_t mark = ws.used;
    const std::uint32_t cap = L.n / (kRuler / 4) + 64;  // generous bound on the ruler count
    // cnt: [0] rulers, [1] the head's ruler, [2] valid nodes, [3] nodes walked,
    // [4] rulers that walks split off
    std::uint32_t* cnt = ws.take<std::uint32_t>(5);
    Rec* rec = ws.take<Rec>(L.n);
    // The ruler count is data dependent; size everything by `cap` and let the
    // kernels read the true count. A count above `cap` is reported.
    std::uint32_t* rulers = ws.take<std::uint32_t>(cap);
    std::uint32_t* nxt = ws.take<std::uint32_t>(cap);
    std::int32_t* sub0 = ws.take<std::int32_t>(cap);
    std::int32_t* sub1 = ws.take<std::int32_t>(cap);
    std::int32_t* P0 = ws.take<std::int32_t>(cap);
    std::int32_t* P1 = ws.take<std::int32_t>(cap);
    std::uint32_t* nhead = cnt + 1;
    if (!cnt || !rec || !rulers || !nxt || !sub0 || !sub1 || !P0 || !P1) return cudaErrorMemoryAllocation;
    cudaMemsetAsync(cnt, 0, sizeof(std::uint32_t) * 5, st);
    ruler_compact<Rec>
        <<<grid_blocks((L.n + kCompactPer - 1) / kCompactPer, 256), 256, 0, st>>>(L, cap, rulers, rec, cnt);
    // Bytes touched per node: successor 4 in, the record out.
    LSDTT_TIMED("stack_ruler_walk", (4.0 + sizeof(Rec)) * static_cast<double>(L.n), st,
                (ruler_walk<Rec><<<grid_blocks(cap, 128), 128, 0, st>>>(L, rulers, cnt, rec, sub0, sub1, nxt, nhead, cap, err)));
    ruler_checks<<<1, 1, 0, st>>>(cnt, cap, err);
    RankLevel up{cap, nxt, sub0, sub1, nullptr, nhead, cnt};
    const cudaError_t e = rank_list(up, P0, P1, ws, err, st);
    if (e != cudaSuccess) return e;
    launch_finish(L, rec, P0, P1, cap, p0, p1, err, st, sv);
    ws.used = mark;
    return cudaGetLastError();
}



// Per-cell s-vector outputs from the two prefix sums (lists short enough for
// the serial ranking).
__global__ void sv_outputs(SvOut o, const std::int32_t* __restrict__ p0, const std::int32_t* __restrict__ p1,
                           unsigned long long* __restrict__ err)
{
    LSDTT_COUNT();
    const std::int64_t c = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= o.g.n || sv_masked(o, c)) return;
    sv_store(o, c, p0[2 * c], p0[2 * c + 1], p1[2 * c], err);
}

// ---- range max over the s-vector: blocks of 32, sparse table over blocks ----
__global__ void rmq_base(const std::int64_t* __restrict__ svec, const std::int32_t* __restrict__ depth,
                         std::int64_t n, std::uint64_t* __restrict__ A, std::uint64_t* __restrict__ pre,
                         std::uint64_t* __restrict__ suf, std::uint64_t* __restrict__ blk)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    std::uint64_t a = 0;
    if (i < n)
    {
        const std::int64_t c = svec[i];
        a = (static_cast<std::uint64_t>(static_cast<std::uint32_t>(depth[c])) << 32) | static_cast<std::uint32_t>(c);
        A[i] = a;
    }
    std::uint64_t p = a;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const std::uint64_t y = __shfl_up_sync(0xffffffffu, p, o);
        if (lane >= o && y > p) p = y;
    }
    std::uint64_t s = a;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const std::uint64_t y = __shfl_down_sync(0xffffffffu, s, o);
        if (lane + o < 32 && y > s) s = y;
    }
    if (i < n)
    {
        pre[i] = p;
        suf[i] = s;
    }
    if (lane == 31 && (i - 31) < n) blk[i >> 5] = p;
}

__global__ void rmq_level(const std::uint64_t* __restrict__ prev, std::int64_t nb, std::int64_t half,
                          std::uint64_t* __restrict__ next)
{
    LSDTT_COUNT();
    const std::int64_t b = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (b >= nb) return;
    std::uint64_t v = prev[b];
    if (b + half < nb && prev[b + half] > v) v = prev[b + half];
    next[b] = v;
}

// All levels of a small table (level k at base + k * stride; level 0 is there)
// by one block, in shared memory: a launch a level took 2.5 us for nothing.
constexpr int kRmqBlock = 4096;

__global__ void __launch_bounds__(1024) rmq_levels(std::uint64_t* __restrict__ base, std::int64_t stride, int nb,
                                                   int levels)
{
    LSDTT_COUNT();
    __shared__ std::uint64_t t[kRmqBlock];
    constexpr int kPer = kRmqBlock / 1024;
    for (int b = threadIdx.x; b < nb; b += 1024) t[b] = base[b];
    __syncthreads();
    for (int k = 1; k < levels; ++k)
    {
        const int half = 1 << (k - 1);
        std::uint64_t v[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j)
        {
            const int b = j * 1024 + threadIdx.x;
            v[j] = b < nb ? t[b] : 0;
            if (b + half < nb && t[b + half] > v[j]) v[j] = t[b + half];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPer; ++j)
        {
            const int b = j * 1024 + threadIdx.x;
            if (b >= nb) continue;
            t[b] = v[j];
            base[k * stride + b] = v[j];
        }
        __syncthreads();
    }
}

struct Rmq
{
    const std::uint64_t* A;
    const std::uint64_t* pre;
    const std::uint64_t* suf;
    const std::uint64_t* table[40];  // the levels, by value
};

__device__ std::uint64_t rmq_query(const Rmq& R, std::int64_t a, std::int64_t b)  // inclusive
{
    const std::int64_t ba = a >> 5, bb = b >> 5;
    if (ba == bb)
    {
        std::uint64_t m = 0;
        for (std::int64_t i = a; i <= b; ++i)
            if (R.A[i] > m) m = R.A[i];
        return m;
    }
    std::uint64_t m = R.suf[a];
    if (R.pre[b] > m) m = R.pre[b];
    const std::int64_t lo = ba + 1, hi = bb - 1;
    if (lo <= hi)
    {
        const std::int64_t len = hi - lo + 1;
        const int k = 63 - __clzll(static_cast<unsigned long long>(len));
        const std::uint64_t* T = R.table[k];
        std::uint64_t x = T[lo];
        const std::uint64_t y = T[hi - (std::int64_t(1) << k) + 1];
        if (y > x) x = y;
        if (x > m) m = x;
    }
    return m;
}

constexpr int kHeightPer = 4;  // cells per thread of topo_heights

// Height and deepest headwater of cell c; returns the height (0: masked).
__device__ __forceinline__ unsigned topo_height(std::int64_t c, const std::uint8_t* __restrict__ mask,
                                                const std::int64_t* __restrict__ start,
                                                const std::uint64_t* __restrict__ size,
                                                const std::int32_t* __restrict__ depth, const Rmq& R,
                                                std::int32_t* __restrict__ height, std::uint32_t* __restrict__ leaf)
{
    if (!mask[c])
    {
        height[c] = -1;
        return 0;
    }
    const std::int64_t a = start[c];
    const std::int64_t s = static_cast<std::int64_t>(size[c]);
    if (a < 0 || s <= 1)
    {
        // a headwater is its own deepest cell (about half of the cells); a
        // cell outside the tour was reported by sv_outputs
        height[c] = 0;
        leaf[c] = static_cast<std::uint32_t>(c);
        return 0;
    }
    const std::uint64_t m = rmq_query(R, a, a + s - 1);
    const std::int32_t h = static_cast<std::int32_t>(m >> 32) - depth[c];
    height[c] = h;
    leaf[c] = static_cast<std::uint32_t>(m & 0xffffffffull);
    return static_cast<unsigned>(h);
}

// The tallest level by one atomic a block: one a warp queued up on its address
// (16.4 M cells 492 us, now 247). Every thread takes part in the warp's
// maximum, whatever its cell.
__global__ void __launch_bounds__(256) topo_heights(Grid g, const std::uint8_t* __restrict__ mask,
                                                    const std::int64_t* __restrict__ start,
                                                    const std::uint64_t* __restrict__ size,
                                                    const std::int32_t* __restrict__ depth, Rmq R,
                                                    std::int32_t* __restrict__ height,
                                                    std::uint32_t* __restrict__ leaf,
                                                    unsigned long long* __restrict__ maxh)
{
    LSDTT_COUNT();
    __shared__ unsigned wmax[8];
    const std::int64_t base = static_cast<std::int64_t>(blockIdx.x) * (256 * kHeightPer) + threadIdx.x;
    unsigned h = 0;
    for (int k = 0; k < kHeightPer; ++k)
    {
        const std::int64_t c = base + 256 * k;
        if (c < g.n) h = max(h, topo_height(c, mask, start, size, depth, R, height, leaf));
    }
    h = __reduce_max_sync(0xffffffffu, h);
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = h;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (int w = 1; w < 8; ++w) h = max(h, wmax[w]);
        if (h) atomicMax(maxh, static_cast<unsigned long long>(h));
    }
}

// Sort keys (height, headwater); invalid cells get height maxh+1 so they
// sort after every valid cell and are dropped.
__global__ void topo_keys(Grid g, const std::uint8_t* __restrict__ mask, const std::int32_t* __restrict__ height,
                          const std::uint32_t* __restrict__ leaf, int leaf_bits, std::uint64_t maxh,
                          std::uint64_t* __restrict__ keys, std::uint32_t* __restrict__ vals)
{
    LSDTT_COUNT();
    const std::int64_t c = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= g.n) return;
    const std::uint64_t h = mask[c] ? static_cast<std::uint64_t>(height[c]) : maxh + 1;
    const std::uint64_t l = mask[c] ? leaf[c] : 0u;
    keys[c] = (h << leaf_bits) | l;
    vals[c] = static_cast<std::uint32_t>(c);
}

__global__ void topo_store(const std::uint32_t* __restrict__ vals, std::int64_t n_valid, std::int64_t* __restrict__ topo,
                           std::uint32_t* __restrict__ topo_pos)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n_valid) return;
    const std::uint32_t c = vals[i];
    topo[i] = c;
    topo_pos[c] = static_cast<std::uint32_t>(i);
}

int bits_for(std::uint64_t v)
{
    int b = 0;
    while (v) { ++b; v >>= 1; }
    return b;
}

}  // namespace

cudaError_t build_stack(lsdtt_gpu_flow* f, bool want_topo, cudaStream_t st, const Packed* packed)
{
    const Grid& g = f->g;
    const std::int64_t n = g.n;
    Scratch& ws = f->ws;
    const std::size_t mark = ws.used;
    const unsigned nb = grid_blocks(n, 256);

    std::uint32_t* first_child = ws.take<std::uint32_t>(n);
    std::uint32_t* next_sib = ws.take<std::uint32_t>(n);
    std::uint32_t* succ = ws.take<std::uint32_t>(2 * n);
    std::uint32_t* head = ws.take<std::uint32_t>(1);
    // A tour longer than kSerialLimit writes the s-vector outputs straight
    // from the ruler records; only the serial ranking needs prefix arrays.
    const bool fused = 2 * n > kSerialLimit;
    std::int32_t* p0 = fused ? nullptr : ws.take<std::int32_t>(2 * n);
    std::int32_t* p1 = fused ? nullptr : ws.take<std::int32_t>(2 * n);
    if (!first_child || !next_sib || !succ || !head || (!fused && (!p0 || !p1))) return cudaErrorMemoryAllocation;

    if (packed)
    {
        if (want_topo) return cudaErrorInvalidValue;  // the ensemble needs the s-vector only
        links_packed<<<nb, 256, 0, st>>>(*packed, f->mask, f->dir, first_child, next_sib);
    }
    else
        links_kernel<<<nb, 256, 0, st>>>(g, f->mask, f->dir, first_child, next_sib);
    root_links_kernel<<<std::min(nb, 152u * 8u), 256, 0, st>>>(f->outlets, f->dscal + 1, next_sib, head);
    succ_kernel<<<nb, 256, 0, st>>>(g, f->mask, f->receiver, first_child, next_sib, succ);

    RankLevel L0{static_cast<std::uint32_t>(2 * n), succ, nullptr, nullptr, f->mask, head, nullptr};
    // The ensemble reads the counts and depths only.
    const SvOut sv{g,          f->mask, f->n_valid, packed ? nullptr : f->sv_start, f->sv_size, f->depth,
                   packed ? nullptr : f->svec};
    cudaError_t e = rank_list(L0, p0, p1, ws, f->derr, st, fused ? &sv : nullptr);
    if (e != cudaSuccess) return e;
    if (!fused) sv_outputs<<<nb, 256, 0, st>>>(sv, p0, p1, f->derr);
    ws.used = mark;  // tour buffers are no longer needed
    if (!want_topo) return cudaGetLastError();

    // Range-max structure over the s-vector.
    const std::int64_t nv = f->n_valid;
    if (nv == 0) return cudaGetLastError();
    const std::int64_t nblk = (nv + 31) / 32;
    std::uint64_t* A = ws.take<std::uint64_t>(nv);
    std::uint64_t* pre = ws.take<std::uint64_t>(nv);
    std::uint64_t* suf = ws.take<std::uint64_t>(nv);
    int levels = 1;
    while ((std::int64_t(1) << levels) <= nblk) ++levels;
    const std::int64_t stride = (nblk + 31) / 32 * 32;
    std::uint64_t* tab = ws.take<std::uint64_t>(static_cast<std::size_t>(stride) * levels);
    if (!A || !pre || !suf || !tab || levels > 40) return cudaErrorMemoryAllocation;
    rmq_base<<<grid_blocks(nblk * 32, 256), 256, 0, st>>>(f->svec, f->depth, nv, A, pre, suf, tab);
    if (nblk <= kRmqBlock)
        rmq_levels<<<1, 1024, 0, st>>>(tab, stride, static_cast<int>(nblk), levels);
    else
        for (int k = 1; k < levels; ++k)
            rmq_level<<<grid_blocks(nblk, 256), 256, 0, st>>>(tab + (k - 1) * stride, nblk, std::int64_t(1) << (k - 1),
                                                              tab + k * stride);

    std::uint64_t* k0 = ws.take<std::uint64_t>(n);
    std::uint32_t* v0 = ws.take<std::uint32_t>(n);
    std::uint64_t* k1 = ws.take<std::uint64_t>(n);
    std::uint32_t* v1 = ws.take<std::uint32_t>(n);
    std::uint32_t* leaf = ws.take<std::uint32_t>(n);
    if (!k0 || !v0 || !k1 || !v1 || !leaf) return cudaErrorMemoryAllocation;
    const int leaf_bits = bits_for(static_cast<std::uint64_t>(n - 1) | 1);
    Rmq R{A, pre, suf, {}};
    for (int k = 0; k < levels; ++k) R.table[k] = tab + k * stride;
    cudaMemsetAsync(f->derr + 2, 0, sizeof(unsigned long long), st);
    topo_heights<<<grid_blocks(n, 256 * kHeightPer), 256, 0, st>>>(g, f->mask, f->sv_start, f->sv_size, f->depth, R, f->height, leaf, f->derr + 2);
    // The number of radix passes depends on the tallest level: read it back.
    cudaMemcpyAsync(&f->herr[2], f->derr + 2, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
    e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    const std::uint64_t maxh = f->herr[2];
    f->max_height = static_cast<std::int64_t>(maxh);
    topo_keys<<<nb, 256, 0, st>>>(g, f->mask, f->height, leaf, leaf_bits, maxh, k0, v0);
    const int bits = leaf_bits + bits_for(maxh + 1);
    const int cur = radix_sort_pairs(k0, v0, k1, v1, n, bits, ws, st, &e);
    if (e != cudaSuccess) return e;
    topo_store<<<grid_blocks(nv, 256), 256, 0, st>>>(cur ? v1 : v0, nv, f->topo, f->topo_pos);
    ws.used = mark;
    return cudaGetLastError();
}


// ---------------------------------------------------------------------------
// accumulate (src/cpu/lsdtt_flowinfo_cpu.cpp:1979-2046)
//
// The reference seeds every valid cell with its weight and pushes
// acc[rec] += acc[flat] in topological order, so a receiver's total is its
// weight plus its donors' totals added in the donors' topological order.
// When every partial sum is exactly representable (default weights dx^2 with
// dx^2 = m*2^e and n_valid*m < 2^53) the order cannot matter and the total is
// size*dx^2 exactly: one pass. Otherwise the totals are formed level by level
// (height 0 first) with each cell adding its donors in topological order --
// the reference's additions in the reference's order.
// ---------------------------------------------------------------------------
namespace
{

__global__ void accum_exact(Grid g, const std::uint8_t* __restrict__ mask, const std::uint64_t* __restrict__ size,
                            double w, double* __restrict__ out)
{
    LSDTT_COUNT();
    const std::int64_t c = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= g.n) return;
    out[c] = mask[c] ? static_cast<double>(size[c]) * w : 0.0;
}

__global__ void accum_seed(Grid g, const std::uint8_t* __restrict__ mask, const double* __restrict__ w, double dw,
                           double* __restrict__ out)
{
    LSDTT_COUNT();
    const std::int64_t c = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c >= g.n) return;
    out[c] = mask[c] ? (w ? w[c] : dw) : 0.0;
}

// A cell's donors in topological order, as one word: their number (bits 0-3)
// and 3 bits of direction each, and whether it is on the grid's edge. It is formed for all cells at once, so a level
// waits for its additions only, not for the search, the positions and the sort
// before them.
constexpr std::uint32_t kAccumEdge = 1u << 28;

__global__ void __launch_bounds__(256) accum_codes(Grid g, const std::uint8_t* __restrict__ dir,
                                                   const std::int64_t* __restrict__ topo,
                                                   const std::uint32_t* __restrict__ topo_pos, std::int64_t lo,
                                                   std::int64_t nv, std::uint32_t* __restrict__ code)
{
    LSDTT_COUNT();
    const std::int64_t i = lo + static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    const std::int64_t c = topo[i];
    const int row = static_cast<int>(c / g.nc), col = static_cast<int>(c % g.nc);
    const bool inner = is_interior(g, row, col);
    std::uint64_t key[8];  // position << 3 | direction; all ones: no donor
    unsigned k = 0;
#pragma unroll
    for (int d = 0; d < 8; ++d)
    {
        std::int64_t nf = c + static_cast<std::int64_t>(d8_dr(d)) * g.nc + d8_dc(d);
        if (!inner)
        {
            const Step s = resolve_step(g, row, col, d);
            nf = s.kind == 1 ? static_cast<std::int64_t>(s.r) * g.nc + s.c : c;
        }
        // (a masked cell has no direction, and c's own does not lead to c)
        const bool donor = nf != c && dir[nf] == ((d + 4) & 7);
        key[d] = donor ? (static_cast<std::uint64_t>(topo_pos[nf]) << 3) | static_cast<unsigned>(d) : ~0ull;
        k += donor ? 1u : 0u;
    }
    // odd-even transposition sort of the eight keys, in registers
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int j = r & 1; j + 1 < 8; j += 2)
        {
            const std::uint64_t x = key[j], y = key[j + 1];
            key[j] = x < y ? x : y;
            key[j + 1] = x < y ? y : x;
        }
    std::uint32_t w = k | (inner ? 0u : kAccumEdge);
#pragma unroll
    for (int j = 0; j < 8; ++j) w |= static_cast<std::uint32_t>(key[j] & 7u) << (4 + 3 * j);
    code[i] = w;
}

__device__ __forceinline__ void accum_cell(const Grid& g, std::int64_t c, std::uint32_t w, double* acc)
{
    const int k = static_cast<int>(w & 15u);
    if (k == 0) return;
    double v[8];
    if (w & kAccumEdge)
    {
        const int row = static_cast<int>(c / g.nc), col = static_cast<int>(c % g.nc);
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            if (j >= k) break;
            const Step s = resolve_step(g, row, col, static_cast<int>((w >> (4 + 3 * j)) & 7u));
            v[j] = acc[static_cast<std::int64_t>(s.r) * g.nc + s.c];
        }
    }
    else
    {
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
            if (j >= k) break;
            const int d = static_cast<int>((w >> (4 + 3 * j)) & 7u);
            v[j] = acc[c + static_cast<std::int64_t>(d8_dr(d)) * g.nc + d8_dc(d)];
        }
    }
    double s = acc[c];
#pragma unroll
    for (int j = 0; j < 8; ++j)
    {
        if (j >= k) break;
        s = __dadd_rn(s, v[j]);
    }
    acc[c] = s;
}

__global__ void __launch_bounds__(128) accum_level(Grid g, const std::int64_t* __restrict__ topo,
                                                   const std::uint32_t* __restrict__ code, std::int64_t lo,
                                                   std::int64_t hi, double* acc)
{
    LSDTT_COUNT();
    const std::int64_t i = lo + static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < hi) accum_cell(g, topo[i], code[i], acc);
}

// The levels from k0 on by one block, a barrier between them: a level is no
// wider than the one below it (each of its cells has a donor there), so once a
// level fits the block's few passes all later ones do. The next level's cells
// are fetched while this one adds. 129 x 203 cells, 27 levels: 244 us in 27
// launches, now 75 in two; 2048 cells and reading the level bounds on the device
// only (no launch for the widest levels) were no faster.
constexpr int kAccumTail = 4096;

__global__ void __launch_bounds__(1024) accum_tail(Grid g, const std::int64_t* __restrict__ topo,
                                                   const std::uint32_t* __restrict__ code,
                                                   const std::int64_t* __restrict__ start, std::int64_t k0,
                                                   std::int64_t nlev, double* acc)
{
    LSDTT_COUNT();
    const std::int64_t nv = start[nlev];
    std::int64_t lo = start[k0], hi = start[k0 + 1];
    std::int64_t c = 0;
    std::uint32_t w = 0;
    if (lo + threadIdx.x < nv)
    {
        c = topo[lo + threadIdx.x];
        w = code[lo + threadIdx.x];
    }
    for (std::int64_t k = k0; k < nlev; ++k)
    {
        std::int64_t cn = 0;
        std::uint32_t wn = 0;
        if (hi + threadIdx.x < nv)
        {
            cn = topo[hi + threadIdx.x];
            wn = code[hi + threadIdx.x];
        }
        const std::int64_t next = k + 1 < nlev ? start[k + 2] : hi;
        if (lo + threadIdx.x < hi) accum_cell(g, c, w, acc);
        for (std::int64_t i = lo + 1024 + threadIdx.x; i < hi; i += 1024) accum_cell(g, topo[i], code[i], acc);
        __syncthreads();
        lo = hi;
        hi = next;
        c = cn;
        w = wn;
    }
}

__global__ void level_bounds(const std::int64_t* __restrict__ topo, const std::int32_t* __restrict__ height,
                             std::int64_t nv, std::int64_t* __restrict__ start)
{
    LSDTT_COUNT();
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= nv) return;
    const std::int32_t h = height[topo[i]];
    if (i == 0 || height[topo[i - 1]] != h) start[h] = i;
    if (i == nv - 1) start[h + 1] = nv;
}

bool exact_by_count(double dw, std::int64_t nv)
{
    // dw = m * 2^e with m odd; exact iff nv * m < 2^53.
    if (!(dw > 0.0) || !std::isfinite(dw)) return false;
    int e = 0;
    double fr = std::frexp(dw, &e);  // dw = fr * 2^e, fr in [0.5, 1)
    std::uint64_t m = static_cast<std::uint64_t>(std::ldexp(fr, 53));
    while (m && !(m & 1)) m >>= 1;
    const long double prod = static_cast<long double>(m) * static_cast<long double>(nv);
    return prod < 9007199254740992.0L;
}

}  // namespace

cudaError_t accumulate(lsdtt_gpu_flow* f, const double* w, double* out, cudaStream_t st, bool* exact_path)
{
    const Grid& g = f->g;
    const unsigned nb = grid_blocks(g.n, 256);
    const double dw = g.cell * g.cell;
    if (!w && exact_by_count(dw, f->n_valid))
    {
        *exact_path = true;
        accum_exact<<<nb, 256, 0, st>>>(g, f->mask, f->sv_size, dw, out);
        return cudaGetLastError();
    }
    *exact_path = false;
    accum_seed<<<nb, 256, 0, st>>>(g, f->mask, w, dw, out);
    const std::int64_t nv = f->n_valid;
    if (nv == 0) return cudaGetLastError();
    const std::int64_t nlev = f->max_height + 1;
    Scratch& ws = f->ws;
    const std::size_t mark = ws.used;
    std::int64_t* start = ws.take<std::int64_t>(static_cast<std::size_t>(nlev) + 1);
    std::uint32_t* code = ws.take<std::uint32_t>(static_cast<std::size_t>(nv));
    if (!start || !code) return cudaErrorMemoryAllocation;
    level_bounds<<<grid_blocks(nv, 256), 256, 0, st>>>(f->topo, f->height, nv, start);
    std::int64_t* hstart = static_cast<std::int64_t*>(std::malloc(sizeof(std::int64_t) * (nlev + 1)));
    if (!hstart) return cudaErrorMemoryAllocation;
    cudaMemcpyAsync(hstart, start, sizeof(std::int64_t) * (nlev + 1), cudaMemcpyDeviceToHost, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && nlev > 1)  // level 0 cells have no donors
    {
        const std::int64_t first = hstart[1];
        accum_codes<<<grid_blocks(nv - first, 256), 256, 0, st>>>(g, f->dir, f->topo, f->topo_pos, first, nv, code);
        std::int64_t k = 1;
        for (; k < nlev && hstart[k + 1] - hstart[k] > kAccumTail; ++k)
            accum_level<<<grid_blocks(hstart[k + 1] - hstart[k], 128), 128, 0, st>>>(g, f->topo, code, hstart[k],
                                                                                     hstart[k + 1], out);
        if (k < nlev) accum_tail<<<1, 1024, 0, st>>>(g, f->topo, code, start, k, nlev, out);
    }
    std::free(hstart);
    ws.used = mark;
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace lsdtt_gb300

namespace lsdtt_gb300
{
LSDTT_DEFINE_LAUNCH_READER(stack)
}  // namespace lsdtt_gb300
