// Level kernels and the device-resident tree loop. See grow.cuh.
//
// Reference behaviour each kernel restates (paths within the project):
//   find_kernel + plan_kernel    HistogramNodeSplitFinder::find
//                                (src/split.cpp:101-162,271-297) and
//                                plan_level (src/grower_impl.hpp:212-255)
//   pcount/plan2/pscatter        host_partition (src/step/primitives.hpp:
//                                262-374), demote_empty_splits
//                                (src/grower_impl.hpp:262-298),
//                                commit_children (:303-326)
//   sort/chain                   the column fill's serial cell order
//                                (src/fill/columns.hpp:31-89)
//   subtract_totals_kernel       finish_split (src/step/primitives.hpp:
//                                156-173), Histogram::totals
//                                (include/bonsai/histogram.hpp:84-95),
//                                propagate_monotone_bounds
//                                (src/grower_impl.hpp:52-80)
//   stamp/final kernels          finalize_as_leaf / write_leaf
//                                (src/step/primitives.hpp:42-69)
#include "grow.cuh"

#include <algorithm>
#include <cmath>
#include <functional>
#include <limits>
#include <numeric>
#include <type_traits>

namespace bb
{
namespace
{

constexpr uint32_t k_threads    = 256;
constexpr uint32_t k_part_rows  = 4096; // rows per partition chunk
constexpr uint32_t k_build_rows = 2048; // rows per histogram-build chunk (exact)
constexpr uint32_t k_qbuild_rows = 2048;  // rows per histogram-build chunk (quantised)
constexpr uint32_t k_qctas = 148;        // persistent quantised-histogram CTAs per tile (one per SM)
constexpr uint32_t k_qthreads    = 512;   // threads per quantised-histogram CTA
constexpr uint32_t k_tthreads    = 1024;  // threads per conflict-free (u8) histogram CTA
constexpr uint32_t k_find_thr   = 128;  // threads per (node, feature) find CTA
constexpr uint32_t k_max_bins   = 4096; // per feature, this engine's ceiling
constexpr uint32_t k_exact_bins = 3679; // and the exact form's
constexpr uint32_t k_no_sel_tile = 0xFFFFFFFFu; // an unused slot of a selection's tile table
constexpr uint32_t k_plan_thr   = 512;  // plan kernels: one thread per node

// The walked tree's decision heap (depthwise trees, depth <= 8): slot h's
// children are 2h + 1 and 2h + 2; an entry is x = tile << 8 | position,
// y = split bin | (the missing bin if missing rows go left, else 0xFFFF)
// << 16. The plan kernels fill it as the tree grows (a node carries its
// slot): a split node's entry, and for a leaf above the last level the leaf
// map entry of its leftmost last-level descendant; every other slot keeps
// the always-left entry the tree starts from (split bin 0xFFFF takes every
// code, no tile).
constexpr uint32_t k_no_tile    = 0xFFFFFFu;
constexpr uint32_t k_heap_slots = 255;         // decision slots of a depth-8 heap
constexpr uint32_t k_heap_pass  = 0xFFFFFFFFu; // an always-left entry's y

struct HeapOut
{
    uint2    *heap;    // k_heap_slots entries, or null: no heap for this tree
    uint16_t *leafmap; // 2^depth last-level slots -> leaf node id
    uint32_t  depth;
    uint32_t  per;     // codes per 32-byte mirror tile
};

// y = split bin | (the missing bin when missing rows go left, else 0xFFFF,
// which no code equals) << 16: routes_left is then code <= split bin or code
// == y >> 16, since the split bin is below the missing bin
__device__ __forceinline__ uint2 heap_entry(uint32_t f, uint32_t per, uint32_t split,
                                            uint32_t last, bool dl)
{
    return make_uint2(((f / per) << 8) | (f % per), split | ((dl ? last : 0xFFFFu) << 16));
}

// Slot h holds a leaf: its leftmost last-level descendant names it.
__device__ __forceinline__ void heap_leaf(HeapOut const &ho, uint32_t h, uint32_t id)
{
    uint32_t const lvl = 31 - __clz(h + 1);
    if (ho.heap == nullptr || lvl > ho.depth)
    {
        return;
    }
    if (h < k_heap_slots)
    {
        ho.heap[h] = make_uint2(k_no_tile << 8, k_heap_pass);
    }
    ho.leafmap[((h + 1) << (ho.depth - lvl)) - (1u << ho.depth)] = static_cast<uint16_t>(id);
}

// L2 eviction hints (createpolicy): the mirror's tiles, which a pass reads
// once, are evict-first, so that the arrays every pass of a tree reads again
// (gradient codes, row lists, gradients) stay in L2.
__device__ __forceinline__ uint64_t l2_policy_first()
{
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

__device__ __forceinline__ uint64_t l2_policy_last()
{
    uint64_t p;
    asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// A row's 32 bytes of a mirror tile (32-byte aligned) in one load: two of 16
// bytes looked the sector up twice, and where the first's line had left L1 by
// the second, fetched it twice.
__device__ __forceinline__ void ld_nc_row(uint4 const *src, uint64_t pol, uint4 &a, uint4 &b)
{
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v8.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7}, [%8], %9;"
                 : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z),
                   "=r"(b.w)
                 : "l"(src), "l"(pol));
}

// A 4-byte load with an L2 policy, through the coherent path.
__device__ __forceinline__ uint32_t ld_hint_b32(void const *src, uint64_t pol)
{
    uint32_t v;
    asm volatile("ld.global.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(src), "l"(pol));
    return v;
}

__device__ __forceinline__ uint32_t ld_nc_u16(uint16_t const *src, uint64_t pol)
{
    uint16_t v;
    asm volatile("ld.global.nc.L2::cache_hint.u16 %0, [%1], %2;" : "=h"(v) : "l"(src), "l"(pol));
    return v;
}

__device__ __forceinline__ uint32_t ld_nc_code(uint8_t const *src, uint64_t pol)
{
    uint16_t v;
    asm volatile("ld.global.nc.L2::cache_hint.u8 %0, [%1], %2;" : "=h"(v) : "l"(src), "l"(pol));
    return v;
}

__device__ __forceinline__ uint32_t ld_nc_code(uint16_t const *src, uint64_t pol)
{
    return ld_nc_u16(src, pol);
}

__device__ __forceinline__ uint32_t lanemask_lt()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

template <typename BinT>
__device__ __forceinline__ uint32_t bin_at(void const *bins, uint64_t n_pad, uint32_t f,
                                           uint32_t r)
{
    return static_cast<BinT const *>(bins)[(static_cast<uint64_t>(f) * n_pad) + r];
}

// Block-wide exclusive scan of one value per thread (blockDim <= 1024).
template <uint32_t NT>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t *total)
{
    __shared__ uint32_t warp_sums[NT / 32];
    uint32_t const      lane = threadIdx.x & 31;
    uint32_t const      w    = threadIdx.x >> 5;
    uint32_t            x    = v;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1)
    {
        uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o)
        {
            x += y;
        }
    }
    if (lane == 31)
    {
        warp_sums[w] = x;
    }
    __syncthreads();
    if (w == 0)
    {
        uint32_t s = lane < NT / 32 ? warp_sums[lane] : 0;
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1)
        {
            uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, s, o);
            if (lane >= o)
            {
                s += y;
            }
        }
        if (lane < NT / 32)
        {
            warp_sums[lane] = s;
        }
    }
    __syncthreads();
    uint32_t const before = w > 0 ? warp_sums[w - 1] : 0;
    if (total != nullptr)
    {
        *total = warp_sums[NT / 32 - 1];
    }
    __syncthreads();
    return before + x - v;
}

// True in the block that passes here last of n: its threads then see what the
// others wrote before. (ticket: zero between launches.)
__device__ __forceinline__ bool last_block(uint32_t *ticket, uint32_t n)
{
    __shared__ bool last_s;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        last_s = atomicAdd(ticket, 1u) == n - 1;
        if (last_s)
        {
            *ticket = 0;
            __threadfence();
        }
    }
    __syncthreads();
    return last_s;
}

__device__ __forceinline__ void write_leaf_node(TreeOut const &t, uint32_t id, float v)
{
    t.feature[id]      = k_leaf_flag;
    t.value[id]        = v;
    t.left[id]         = 0;
    t.right[id]        = 0;
    t.default_left[id] = 0;
    t.split_bin[id]    = 0;
}

__device__ __forceinline__ float leaf_value(Node const &nd, TreeParams const &tp)
{
    return static_cast<float>(bounded_leaf_weight(nd.sum_g, nd.sum_h, tp.lambda_l1,
                                                  tp.lambda_l2, nd.lo, nd.hi));
}

// ---------------------------------------------------------------- root ----

// n_root_dev (nullable): the root's row count lives on the device (a row
// sample drawn for this tree); an unsharded root's global count is then the
// same number.
} // namespace

struct RootArgs
{
    Ctl            *ctl;
    Node           *nodes;
    uint32_t        n_root;
    Chunk          *bchunks;
    uint32_t       *brange;
    uint32_t       *build;
    TreeOut         t;
    uint32_t        crows;
    uint32_t        g_root;
    uint32_t const *n_root_dev;
    uint2          *heap;
};

namespace
{

__device__ __forceinline__ void root_setup(RootArgs const &A)
{
    Ctl *const            ctl        = A.ctl;
    Node *const           nodes      = A.nodes;
    uint32_t              n_root     = A.n_root;
    Chunk *const          bchunks    = A.bchunks;
    uint32_t *const       brange     = A.brange;
    uint32_t *const       build      = A.build;
    TreeOut const        &t          = A.t;
    uint32_t const        crows      = A.crows;
    uint32_t              g_root     = A.g_root;
    uint32_t const *const n_root_dev = A.n_root_dev;
    uint2 *const          heap       = A.heap;
    for (uint32_t i = threadIdx.x; heap != nullptr && i < k_heap_slots; i += blockDim.x)
    {
        heap[i] = make_uint2(k_no_tile << 8, k_heap_pass);
    }
    if (n_root_dev != nullptr)
    {
        n_root = *n_root_dev;
        g_root = n_root;
    }
    uint32_t const nch = (n_root + crows - 1) / crows;
    if (threadIdx.x == 0)
    {
        Ctl c{};
        c.n_cur      = 1;
        c.n_nodes    = 1;
        c.n_build    = 1;
        c.n_bchunks  = nch;
        c.built_rows = n_root;
        *ctl         = c;
        Node nd{};
        nd.start  = 0;
        nd.count  = n_root;
        nd.gcount = g_root;
        nd.id     = 0;
        nd.lo     = -INFINITY;
        nd.hi     = INFINITY;
        nodes[0]  = nd;
        build[0]  = 0;
        brange[0] = 0;
        brange[1] = nch;
        write_leaf_node(t, 0, 0.0F);
        t.gain[0]  = 0.0F;
        t.cover[0] = static_cast<float>(g_root);
    }
    for (uint32_t c = threadIdx.x; c < nch; c += blockDim.x)
    {
        uint32_t const b = c * crows;
        bchunks[c]       = {0, b, min(crows, n_root - b), 0};
    }
}

__global__ void root_setup_kernel(RootArgs A)
{
    pdl_enter();
    root_setup(A);
}

// The next 32 terms of a warp's serial FP64 sum, in order: lane i holds term i
// (0 past the end, which leaves the sum as it is: it starts at +0 and so is
// never -0), every lane adds them all and keeps the sum at its own. The chain is
// one dependent add a term; the shuffles that feed it run ahead. (One thread
// that read, added and wrote a cell at a time took 40 ns a bin; of a level of
// 20,640 rows x 8 the find 14.7 us and the totals 14.7 before, 10.6 and 9.3 now, under ncu.)
__device__ __forceinline__ double warp_serial_sum(double term, double &sum)
{
    uint32_t const lane = threadIdx.x & 31;
    double         mine = 0.0;
#pragma unroll
    for (uint32_t i = 0; i < 32; ++i)
    {
        sum += __shfl_sync(0xFFFFFFFFu, term, i);
        mine = lane == i ? sum : mine;
    }
    return mine;
}

// Node totals from the first selected feature's cells: double sums over
// every cell in bin order, rounded to float once (Histogram::totals), with
// one warp, each lane holding them.
template <typename Cells>
__device__ __forceinline__ void warp_totals(Cells const &cells, uint32_t nb, float &g, float &h)
{
    uint32_t const lane = threadIdx.x & 31;
    double         sg   = 0.0;
    double         sh   = 0.0;
    for (uint32_t b0 = 0; b0 < nb; b0 += 32)
    {
        float2 const c = b0 + lane < nb ? cells(b0 + lane) : make_float2(0.0F, 0.0F);
        warp_serial_sum(c.x, sg);
        warp_serial_sum(c.y, sh);
    }
    g = static_cast<float>(sg);
    h = static_cast<float>(sh);
}

__global__ void root_totals_kernel(Node *nodes, float2 const *hist, uint32_t const *sel_nb)
{
    pdl_enter();
    float g, h;
    warp_totals([&](uint32_t b) { return hist[b]; }, sel_nb[0], g, h);
    if (threadIdx.x == 0)
    {
        nodes[0].sum_g = g;
        nodes[0].sum_h = h;
    }
}

// ------------------------------------------------------- histogram build ----
// The plain form's cells must equal the CPU fill's serial float chains: each
// cell's (g, h) values added one by one in the node's row order. Two kernels:
//
// sort_kernel: a CTA takes one 2,048-row chunk of a built node and one mirror
// tile, brings each row's 32-byte tile and gradient pair into shared memory
// once, and counting-sorts the rows by bin, stably, feature after feature
// (four features at a time, a group of four warps each). A node of one chunk
// is finished here, a thread per bin adding its run; the others' sorted pairs
// go to memory, coalesced, with the chunk's bin offsets.
//
// chain_kernel: a warp takes 32 bins of a (node, feature), a lane per bin, and
// streams that range of the node's chunks in order through a shared-memory
// ring, each lane adding its runs.
//
// A bin's run is an even number of pairs, an odd one ending with a pair of
// +0.0: two pairs are then one aligned 16-byte read. Adding +0.0 changes
// nothing -- a sum that starts at +0.0 is never -0.0 under round-to-nearest.
//
// A chunk is sorted on its own: no counting pass over the node comes first,
// rows and tiles are read once for all of a tile's features, and the payload
// is written and read in whole lines. The former form -- a counting pass, a
// per-node offset pass, a scatter of single pairs to 256 open places per
// feature and a chain reading one line per lane -- took 32.7 ms per tree of
// the 10M x 28 depth-8 logloss fit; these two take 11.5 (sort 6.6, bound by
// the integer pipe's ballots; chain 4.9, by the largest nodes' serial chains).

constexpr uint32_t k_xgthr   = 128; // a group: one feature at a time
constexpr uint32_t k_xgwarps = k_xgthr / 32;
constexpr uint32_t k_xsteps  = k_build_rows / k_xgthr; // rows per lane and feature
constexpr uint32_t k_xgroups = 4;  // groups per CTA, where their tables fit
static_assert(2 * k_build_rows <= 0x1000, "a place in a padded chunk takes 12 bits");

// A group's barrier (barrier 0 is the CTA's).
__device__ __forceinline__ void group_sync(uint32_t group)
{
    asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(k_xgthr) : "memory");
}

// Adds a pair to a pair: two IEEE float adds in one instruction.
__device__ __forceinline__ void add_pair(float2 &a, float2 const b)
{
    auto      &x = reinterpret_cast<unsigned long long &>(a);
    auto const y = reinterpret_cast<unsigned long long const &>(b);
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(x) : "l"(y));
}

// 16-bit words of a chunk's offset row: its bins in whole warps of 32, the
// end after the last one, and room to keep rows 16-byte aligned.
__host__ __device__ inline uint32_t offset_stride(uint32_t max_nb)
{
    return (((max_nb + 31) / 32) * 32) + 8;
}

// Pairs that padding may add to a chunk (even).
__host__ __device__ inline uint32_t chunk_pads(uint32_t max_nb)
{
    return (min(max_nb, k_build_rows) + 1) & ~1u;
}

// Where chunk c (the x-th of its node, whose rows begin at base among the
// built rows) has its sorted pairs: its rows' place, rounded down to a whole
// 16 bytes, after every earlier chunk's padding.
__device__ __forceinline__ uint64_t chunk_at(uint32_t base, uint32_t x, uint32_t c,
                                             uint32_t max_nb)
{
    return ((uint64_t{base} + (uint64_t{x} * k_build_rows)) & ~uint64_t{1}) +
           (uint64_t{c} * (chunk_pads(max_nb) + 2));
}

// Bytes of sort_kernel's dynamic shared memory.
inline size_t sort_smem(uint32_t max_nb, uint32_t groups)
{
    size_t const row = ((max_nb + 1) / 2) * 4; // one warp's counters, 16 bits a bin
    return (size_t{k_build_rows} * (k_mirror_bytes + sizeof(float2))) + 16 +
           (groups * ((size_t{k_build_rows + chunk_pads(max_nb)} * 2) + (k_xgwarps * row)));
}

// Ranks a warp's rows within their bins, in row order: key[st] is the code of
// the lane's row of step st (0xFFFF: none) and leaves with its rank -- the
// rows before it in its bin, in this warp's run -- in its high half; cnt16
// leaves holding each bin's rows. The lanes of one bin are found from a
// ballot per bit of the code: the match instruction takes about 59 cycles of
// an SM a warp here (root sort of 10M rows 2,509 us with it, 1,384 with the
// ballots, which the integer pipe bounds).
template <uint32_t BITS>
__device__ __forceinline__ void rank_rows(uint32_t (&key)[k_xsteps], uint16_t *cnt16)
{
#pragma unroll
    for (uint32_t st = 0; st < k_xsteps; ++st)
    {
        uint32_t const b     = key[st];
        bool const     valid = b != 0xFFFFu;
        uint32_t       peers = __ballot_sync(0xFFFFFFFFu, valid);
#pragma unroll
        for (uint32_t i = 0; i < BITS; ++i)
        {
            uint32_t const bit = (b >> i) & 1u;
            peers &= __ballot_sync(0xFFFFFFFFu, bit != 0) ^ (bit - 1u);
        }
        uint32_t const lt  = __popc(peers & lanemask_lt());
        uint32_t       old = 0;
        if (valid)
        {
            old = cnt16[b];
        }
        __syncwarp();
        if (valid && lt == 0)
        {
            cnt16[b] = static_cast<uint16_t>(old + __popc(peers));
        }
        __syncwarp();
        key[st] = b | ((old + lt) << 16);
    }
}

// grid (chunks, tiles, parts of a tile's features)
template <typename BinT, uint32_t GROUPS>
__global__ void __launch_bounds__(GROUPS *k_xgthr, GROUPS == k_xgroups && sizeof(BinT) == 1 ? 2 : 1)
    sort_kernel(Ctl const *ctl, Chunk const *bchunks, uint32_t const *brange,
                uint32_t const *build, uint32_t const *__restrict__ rows,
                uint4 const *__restrict__ mirror, uint64_t n_rows,
                float2 const *__restrict__ gh, uint32_t const *tile_ids, int32_t const *tile_j,
                uint32_t const *sel_nb, uint32_t const *cell_off, uint32_t max_nb, uint32_t nfb,
                uint16_t *__restrict__ coff, uint32_t cs, float2 *__restrict__ payload,
                uint64_t p_stride, float2 *hist, uint32_t total_cells)
{
    pdl_enter();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr uint32_t per = k_mirror_bytes / sizeof(BinT);
    uint32_t const     c   = blockIdx.x;
    if (c >= ctl->n_bchunks)
    {
        return;
    }
    uint32_t const tile = tile_ids[blockIdx.y];
    if (tile == k_no_sel_tile)
    {
        return;
    }
    uint32_t const crow   = (max_nb + 1) / 2; // counter words per warp
    uint32_t const orow   = k_build_rows + chunk_pads(max_nb);
    auto          *gh_s   = reinterpret_cast<float2 *>(smem_raw); // [rows], a pair of zeros
    auto          *tile_s = reinterpret_cast<uint32_t *>(gh_s + k_build_rows + 2); // [8 words][rows]
    auto          *cnt_0  = tile_s + (8 * k_build_rows);
    uint32_t const group  = threadIdx.x / k_xgthr;
    uint32_t const gt     = threadIdx.x % k_xgthr;
    uint32_t const wg     = gt / 32;
    uint32_t const lane   = threadIdx.x & 31;
    auto          *cnt_s  = cnt_0 + (group * k_xgwarps * crow); // [warp][bin], 16 bits each
    auto          *order_s =
        reinterpret_cast<uint16_t *>(cnt_0 + (GROUPS * k_xgwarps * crow)) + (group * orow);
    __shared__ uint32_t wsum_s[GROUPS][k_xgwarps];

    Chunk const    ch  = bchunks[c];
    uint32_t const c0  = brange[ch.node];
    bool const     one = brange[ch.node + 1] - c0 == 1;
    for (uint32_t k = threadIdx.x; k < ch.count; k += GROUPS * k_xgthr)
    {
        uint32_t const r  = rows[ch.begin + k];
        uint4 const   *tp = mirror + (((uint64_t{tile} * n_rows) + r) * 2);
        uint4 const    lo = __ldg(tp);
        uint4 const    hi = __ldg(tp + 1);
        gh_s[k]           = __ldg(gh + r);
        // a plane per 4-byte word, so that a feature's codes of consecutive
        // rows lie in consecutive banks
        tile_s[k]                      = lo.x;
        tile_s[k_build_rows + k]       = lo.y;
        tile_s[(2 * k_build_rows) + k] = lo.z;
        tile_s[(3 * k_build_rows) + k] = lo.w;
        tile_s[(4 * k_build_rows) + k] = hi.x;
        tile_s[(5 * k_build_rows) + k] = hi.y;
        tile_s[(6 * k_build_rows) + k] = hi.z;
        tile_s[(7 * k_build_rows) + k] = hi.w;
    }
    if (threadIdx.x == 0)
    {
        gh_s[k_build_rows] = make_float2(0.0F, 0.0F);
    }
    __syncthreads();
    auto          *cnt16 = reinterpret_cast<uint16_t *>(cnt_s + (wg * crow));
    auto const    *start = reinterpret_cast<uint16_t const *>(cnt_s); // after the scan
    uint32_t const k0    = wg * (k_xsteps * 32);
    for (uint32_t x = group + (GROUPS * blockIdx.z); x < per; x += GROUPS * gridDim.z)
    {
        int32_t const js = tile_j[(blockIdx.y * per) + x];
        if (js < 0)
        {
            continue;
        }
        uint32_t const j  = static_cast<uint32_t>(js);
        uint32_t const nb = sel_nb[j];
        for (uint32_t b = lane; b < crow; b += 32)
        {
            cnt_s[(wg * crow) + b] = 0;
        }
        __syncwarp();
        auto const *codes =
            reinterpret_cast<unsigned char const *>(tile_s + ((x * sizeof(BinT) / 4) * k_build_rows)) +
            ((x * sizeof(BinT)) % 4);
        uint32_t key[k_xsteps];
#pragma unroll
        for (uint32_t st = 0; st < k_xsteps; ++st)
        {
            uint32_t const k = k0 + (st * 32) + lane;
            key[st]          = k < ch.count
                                   ? *reinterpret_cast<BinT const *>(codes + (size_t{k} * 4))
                                   : 0xFFFFu;
        }
        // as many ballots as the feature's codes have bits (a uniform choice)
        if (nb <= 16)
        {
            rank_rows<4>(key, cnt16);
        }
        else if (sizeof(BinT) == 1 || nb <= 256)
        {
            rank_rows<8>(key, cnt16);
        }
        else
        {
            rank_rows<12>(key, cnt16);
        }
        group_sync(group);
        // the chunk's (padded) bin starts, and each warp's place in each bin
        uint32_t carry = 0;
        for (uint32_t p0 = 0; p0 < crow; p0 += k_xgthr)
        {
            uint32_t const p = p0 + gt;
            uint32_t       v[k_xgwarps];
            uint32_t       pair = 0; // two bins' counts, 16 bits each
#pragma unroll
            for (uint32_t w = 0; w < k_xgwarps; ++w)
            {
                v[w] = p < crow ? cnt_s[(w * crow) + p] : 0;
                pair += v[w];
            }
            uint32_t const even = (pair + 0x00010001u) & 0xFFFEFFFEu;
            uint32_t const both = (even & 0xFFFFu) + (even >> 16);
            uint32_t       inc  = both;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1)
            {
                uint32_t const y = __shfl_up_sync(0xFFFFFFFFu, inc, o);
                if (lane >= o)
                {
                    inc += y;
                }
            }
            if (lane == 31)
            {
                wsum_s[group][wg] = inc;
            }
            group_sync(group);
            uint32_t before = carry + inc - both;
#pragma unroll
            for (uint32_t w = 0; w < k_xgwarps; ++w)
            {
                uint32_t const t = wsum_s[group][w];
                before += w < wg ? t : 0;
                carry += t;
            }
            // (both halves stay below 2^13: no carry between them)
            uint32_t const second = before + (even & 0xFFFFu);
            uint32_t       run    = before | (second << 16);
            if (p < crow)
            {
#pragma unroll
                for (uint32_t w = 0; w < k_xgwarps; ++w)
                {
                    cnt_s[(w * crow) + p] = run;
                    run += v[w];
                }
                if ((pair & 1u) != 0)
                {
                    order_s[second - 1] = k_build_rows;
                }
                if ((pair & 0x10000u) != 0)
                {
                    order_s[before + both - 1] = k_build_rows;
                }
            }
            group_sync(group);
        }
#pragma unroll
        for (uint32_t st = 0; st < k_xsteps; ++st)
        {
            uint32_t const b = key[st] & 0xFFFFu;
            if (b != 0xFFFFu)
            {
                order_s[cnt16[b] + (key[st] >> 16)] =
                    static_cast<uint16_t>(k0 + (st * 32) + lane);
            }
        }
        group_sync(group);
        // (warp 0's counters are the bins' starts, carry the padded length)
        if (one)
        {
            float2 *cells = hist + (static_cast<uint64_t>(build[ch.node]) * total_cells) + cell_off[j];
            for (uint32_t b = gt; b < nb; b += k_xgthr)
            {
                uint32_t const s1 = b + 1 < nb ? start[b + 1] : carry;
                float2         a  = make_float2(0.0F, 0.0F);
#pragma unroll 2
                for (uint32_t p = start[b]; p < s1; p += 2)
                {
                    uint32_t const two = *reinterpret_cast<uint32_t const *>(order_s + p);
                    add_pair(a, gh_s[two & 0xFFFFu]);
                    add_pair(a, gh_s[two >> 16]);
                }
                cells[b] = a;
            }
        }
        else
        {
            float2 *out = payload + (j * p_stride) + chunk_at(ch.aux, c - c0, c, max_nb);
#pragma unroll 4
            for (uint32_t p = gt; p < carry; p += k_xgthr)
            {
                out[p] = gh_s[order_s[p]];
            }
            uint16_t      *off = coff + (((uint64_t{c} * nfb) + j) * cs);
            uint32_t const end = (((nb + 31) / 32) * 32) + 1;
            for (uint32_t b = gt; b < end; b += k_xgthr)
            {
                off[b] = b < nb ? start[b] : static_cast<uint16_t>(carry);
            }
        }
        group_sync(group);
    }
}

__device__ __forceinline__ void cp_async16(void *smem_dst, void const *gsrc)
{
    uint32_t const s = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gsrc));
}
__device__ __forceinline__ void cp_async_commit()
{
    asm volatile("cp.async.commit_group;\n" ::);
}
template <int N> __device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

// A piece of a chunk's range of 32 bins: at most k_piece pairs (a chunk of
// evenly spread codes has 272 in 32 of 256 bins, so one piece a chunk; a bin
// holding most rows takes several), in one of k_pslots ring slots.
constexpr uint32_t k_piece    = 512;
constexpr uint32_t k_pslots   = 6;
constexpr uint32_t k_plag     = 4;  // copies under way before the oldest is handed over
constexpr uint32_t k_cthreads = 64; // the adding warp and the copying one

// Named barriers of the ring (0 is the CTA's): slot s is full, slot s is empty.
__device__ __forceinline__ void ring_arrive(uint32_t id)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(k_cthreads) : "memory");
}
__device__ __forceinline__ void ring_sync(uint32_t id)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(k_cthreads) : "memory");
}

// grid (build nodes, features, ceil(max_bins / 32)). A level's time is that
// of its largest node, whose chain of chunks is serial, so what counts is a
// chunk's time in the adding warp: a second warp does all of the copying.
__global__ void __launch_bounds__(k_cthreads)
    chain_kernel(Ctl const *ctl, uint32_t const *build, Chunk const *bchunks,
                 uint32_t const *brange, uint16_t const *__restrict__ coff,
                 float2 const *__restrict__ payload, uint64_t p_stride, uint32_t const *sel_nb,
                 uint32_t const *cell_off, uint32_t max_nb, uint32_t nfb, uint32_t cs,
                 float2 *hist, uint32_t total_cells)
{
    pdl_enter();
    __shared__ __align__(16) float2 ring_s[k_pslots][k_piece];
    // a slot's piece: first pair within the chunk | pairs << 12 | the chunk's
    // last piece << 31
    __shared__ uint32_t head_s[k_pslots];
    uint32_t const      i = blockIdx.x;
    if (i >= ctl->n_build)
    {
        return;
    }
    uint32_t const c0 = brange[i];
    uint32_t const c1 = brange[i + 1];
    uint32_t const j  = blockIdx.y;
    uint32_t const nb = sel_nb[j];
    uint32_t const z  = blockIdx.z * 32;
    if (c1 - c0 == 1 || z >= nb)
    {
        return; // one chunk: the sort finished it
    }
    uint32_t const  lane = threadIdx.x & 31;
    size_t const    step = size_t{nfb} * cs;
    uint16_t const *off  = coff + (((uint64_t{c0} * nfb) + j) * cs) + z;
    constexpr uint32_t full  = 1;
    constexpr uint32_t empty = 1 + k_pslots;
    if (threadIdx.x >= 32)
    {
        // every chunk is at least one piece, if an empty one
        uint32_t const base   = c1 > c0 ? bchunks[c0].aux : 0;
        float2 const  *mine   = payload + (j * p_stride);
        uint32_t       piece  = 0;
        uint32_t       slot   = 0; // of the piece being issued
        uint32_t       ready  = 0; // of the oldest copy under way
        for (uint32_t cb = c0; cb < c1; cb += 32)
        {
            // the ranges of 32 chunks at a time, a lane each
            uint32_t const m  = min(32u, c1 - cb);
            uint32_t       r0 = 0;
            uint32_t       r1 = 0;
            if (lane < m)
            {
                r0 = off[lane * step];
                r1 = off[(lane * step) + 32];
            }
            off += 32 * step;
            for (uint32_t x = 0; x < m; ++x)
            {
                uint32_t       ip  = __shfl_sync(0xFFFFFFFFu, r0, x);
                uint32_t const end = __shfl_sync(0xFFFFFFFFu, r1, x);
                float2 const  *src = mine + chunk_at(base, cb + x - c0, cb + x, max_nb) + (2 * lane);
                bool           more;
                do
                {
                    uint32_t const len = min(k_piece, end - ip);
                    more               = end - ip > k_piece;
                    if (piece >= k_pslots)
                    {
                        ring_sync(empty + slot);
                    }
                    float2 const *from = src + ip; // runs are even: 16-byte copies
                    float2       *dst  = &ring_s[slot][2 * lane];
#pragma unroll
                    for (uint32_t u = 0; u < k_piece / 64; ++u)
                    {
                        if (2 * ((u * 32) + lane) < len)
                        {
                            cp_async16(dst + (u * 64), from + (u * 64));
                        }
                    }
                    cp_async_commit();
                    if (lane == 0)
                    {
                        head_s[slot] = ip | (len << 12) | (more ? 0u : 1u << 31);
                    }
                    ip += len;
                    slot = slot + 1 == k_pslots ? 0 : slot + 1;
                    if (++piece > k_plag)
                    {
                        cp_async_wait<k_plag>();
                        ring_arrive(full + ready);
                        ready = ready + 1 == k_pslots ? 0 : ready + 1;
                    }
                } while (more);
            }
        }
        cp_async_wait<0>();
        for (uint32_t x = min(piece, k_plag); x > 0; --x)
        {
            ring_arrive(full + ready);
            ready = ready + 1 == k_pslots ? 0 : ready + 1;
        }
        // the adding warp's last hand-backs
        uint32_t at = (slot + k_pslots - (min(piece, k_pslots) % k_pslots)) % k_pslots;
        for (uint32_t x = min(piece, k_pslots); x > 0; --x)
        {
            ring_sync(empty + at);
            at = at + 1 == k_pslots ? 0 : at + 1;
        }
        return;
    }
    off += lane;
    uint32_t left = c1 - c0; // chunks whose offsets have not been asked for
    auto     offs = [&](uint32_t &lo, uint32_t &hi)
    {
        lo = 0;
        hi = 0;
        if (left > 0)
        {
            lo = off[0];
            hi = off[1];
            off += step;
            --left;
        }
    };
    // this lane's run in the current chunk and in the next three
    uint32_t lo[4], hi[4];
#pragma unroll
    for (uint32_t q = 0; q < 4; ++q)
    {
        offs(lo[q], hi[q]);
    }
    // four reads of two pairs; their additions
    auto take = [](float4(&x)[4], float4 const *v, int n)
    {
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            if (2 * q < n)
            {
                x[q] = v[q];
            }
        }
    };
    auto fold = [](float2 &a, float4 const(&x)[4], int n)
    {
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            if (2 * q < n)
            {
                add_pair(a, make_float2(x[q].x, x[q].y));
                add_pair(a, make_float2(x[q].z, x[q].w));
            }
        }
    };
    float2   a    = make_float2(0.0F, 0.0F);
    uint32_t slot = 0;
    // four chunks at a time, so that each one's offsets keep their registers
    // (moving a register waits for the load that fills it)
    for (uint32_t c = c0; c < c1; c += 4)
    {
#pragma unroll
        for (uint32_t p = 0; p < 4; ++p)
        {
            if (c + p >= c1)
            {
                break;
            }
            bool more;
            do
            {
                ring_sync(full + slot);
                uint32_t const head = head_s[slot];
                uint32_t const ip   = head & 0xFFFu;
                uint32_t const len  = (head >> 12) & 0xFFFu;
                more                = (head >> 31) == 0;
                // the run's part in this piece, eight pairs at a time: the
                // next eight are on their way while these are added
                uint32_t const e0 = max(lo[p], ip);
                int            n  = static_cast<int>(min(hi[p], ip + len)) - static_cast<int>(e0);
                float4 const  *v  = reinterpret_cast<float4 const *>(&ring_s[slot][0]) + ((e0 - ip) / 2);
                float4         x[4], y[4];
                take(x, v, n);
                while (__any_sync(0xFFFFFFFFu, n > 8))
                {
                    take(y, v + 4, n - 8);
                    fold(a, x, n);
                    n -= 8;
                    v += 4;
                    if (!__any_sync(0xFFFFFFFFu, n > 8))
                    {
#pragma unroll
                        for (uint32_t q = 0; q < 4; ++q)
                        {
                            x[q] = y[q];
                        }
                        break;
                    }
                    take(x, v + 4, n - 8);
                    fold(a, y, n);
                    n -= 8;
                    v += 4;
                }
                fold(a, x, n);
                ring_arrive(empty + slot);
                slot = slot + 1 == k_pslots ? 0 : slot + 1;
            } while (more);
            offs(lo[p], hi[p]);
        }
    }
    if (z + lane < nb)
    {
        hist[(static_cast<uint64_t>(build[i]) * total_cells) + cell_off[j] + z + lane] = a;
    }
}

// A quantised cell: with cw == 1 (int8 codes) one packed word -- the int32
// gradient sum in the high half (two's complement), the uint32 hessian sum in
// the low half; with cw == 2 (int16 codes, whose sums outgrow 32 bits) two
// words, the int64 gradient sum then the uint64 hessian sum. x counts cells.
__device__ __forceinline__ void qcell(unsigned long long const *h, uint64_t x, uint32_t cw,
                                      int64_t &g, int64_t &hs)
{
    if (cw == 2)
    {
        g  = static_cast<int64_t>(h[2 * x]);
        hs = static_cast<int64_t>(h[(2 * x) + 1]);
    }
    else
    {
        unsigned long long const c = h[x];
        g  = static_cast<int32_t>(static_cast<uint32_t>(c >> 32));
        hs = static_cast<uint32_t>(c);
    }
}

// ------------------------------------------------------------ split find ----

// The per-candidate core of update_best_for_feature_for_node
// (src/split.cpp:55-82,101-162) for one (bin, default_left).
template <typename M>
__device__ __forceinline__ bool candidate_gain(double lg, double lh, M mg, M mh,
                                               double real_g, double real_h, bool dl,
                                               double node_score, TreeParams const &tp,
                                               int mc, double lo, double hi,
                                               double &gain)
{
    double const rg = real_g - lg;
    double const rh = real_h - lh;
    double const gL = lg + (dl ? static_cast<double>(mg) : 0.0);
    double const hL = lh + (dl ? static_cast<double>(mh) : 0.0);
    double const gR = rg + (!dl ? static_cast<double>(mg) : 0.0);
    double const hR = rh + (!dl ? static_cast<double>(mh) : 0.0);
    double const mch = tp.min_child_hess;
    if (hL < mch || hR < mch)
    {
        return false;
    }
    double const l1       = tp.lambda_l1;
    double const l2       = tp.lambda_l2;
    double const children = split_score(gL, hL, l1, l2) + split_score(gR, hR, l1, l2);
    if (mc != 0)
    {
        double const wl = bounded_leaf_weight(gL, hL, l1, l2, lo, hi);
        double const wr = bounded_leaf_weight(gR, hR, l1, l2, lo, hi);
        if (static_cast<double>(mc) * (wr - wl) < 0.0)
        {
            return false;
        }
    }
    gain = children - node_score;
    return true;
}

// Warp reduce of (gain, order): the larger gain, the earlier scan order on a
// tie, so the winner is the serial scan's strict-> first maximum.
__device__ __forceinline__ void warp_best(double &gain, uint32_t &order)
{
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        double const   g2 = __shfl_xor_sync(0xFFFFFFFFu, gain, o);
        uint32_t const o2 = __shfl_xor_sync(0xFFFFFFFFu, order, o);
        if (g2 > gain || (g2 == gain && o2 < order))
        {
            gain  = g2;
            order = o2;
        }
    }
}

// Interaction constraints (allowed_features / propagate_interaction_state,
// src/grower_impl.hpp:114-160). fgroups[f]: the groups containing feature f
// as a bit mask (at most 64 groups). A node may split on f when its path is
// empty, when a group containing its whole path contains f, or when f is the
// path's only feature.
__device__ __forceinline__ bool interaction_allows(Node const &nd, uint64_t const *fgroups,
                                                   uint32_t f)
{
    uint32_t const plen = nd.ipath & 3u;
    return fgroups == nullptr || plen == 0 || (fgroups[f] & nd.icover) != 0 ||
           (plen == 1 && (nd.ipath >> 2) == f);
}

// Both children's path state after the parent splits on f.
__device__ __forceinline__ void interaction_children(Node const &par, uint64_t const *fgroups,
                                                     uint32_t f, Node &L, Node &R)
{
    if (fgroups == nullptr)
    {
        return;
    }
    uint32_t const plen = par.ipath & 3u;
    uint64_t       cover;
    uint32_t       path;
    if (plen == 0)
    {
        cover = fgroups[f];
        path  = 1u | (f << 2);
    }
    else
    {
        cover = par.icover & fgroups[f];
        path  = (plen == 1 && (par.ipath >> 2) == f) ? par.ipath : 2u;
    }
    L.icover = cover;
    R.icover = cover;
    L.ipath  = path;
    R.ipath  = path;
}

// The exact form's find. grid (frontier, n_sel): one CTA of k_find_thr threads per
// (node, feature), the prefix one serial FP64 chain (the reference's summation
// order), then each thread a few candidates.
__global__ void __launch_bounds__(k_find_thr)
    find_kernel(Ctl const *ctl, Node const *nodes, void const *hist_v,
                uint32_t total_cells, uint32_t const *cell_off, uint32_t const *sel_nb,
                uint32_t const *sel, uint32_t n_sel, int8_t const *mono, uint32_t n_mono,
                TreeParams tp, Best *cand, uint32_t max_nb, uint32_t const *slot_of,
                uint64_t const *fgroups)
{
    pdl_enter();
    extern __shared__ unsigned char smem_raw[];
    __shared__ double   bg_s[k_find_thr / 32];
    __shared__ uint32_t bo_s[k_find_thr / 32];
    uint32_t const      i = blockIdx.x;
    if (i >= ctl->n_cur)
    {
        return;
    }
    uint32_t const tid  = threadIdx.x;
    uint32_t const lane = tid & 31;
    uint32_t const w    = tid >> 5;
    uint32_t const j    = blockIdx.y;
    auto          *pref = reinterpret_cast<double2 *>(smem_raw);                  // [max_nb]
    auto          *cell = reinterpret_cast<float2 *>(pref + max_nb);              // [max_nb]
    Node const     nd   = nodes[i];
    uint32_t const nb   = sel_nb[j];
    Best           out  = {0.0, j, 0, 1, 0};
    if (nd.gcount < 2 * tp.min_data_in_leaf || nb < 2 ||
        !interaction_allows(nd, fgroups, sel[j]))
    {
        if (tid == 0)
        {
            cand[(i * n_sel) + j] = out;
        }
        return;
    }
    uint32_t const n_cut = nb - 2;
    // a node's slot is its frontier index unless slot_of names it (the
    // leafwise pool)
    uint32_t const slot = slot_of != nullptr ? slot_of[i] : i;
    auto const    *src  = static_cast<float2 const *>(hist_v) +
                      ((static_cast<uint64_t>(slot) * total_cells) + cell_off[j]);
    for (uint32_t b = tid; b < nb; b += k_find_thr)
    {
        cell[b] = src[b];
    }
    __syncthreads();
    double const l1 = tp.lambda_l1;
    double const l2 = tp.lambda_l2;
    if (w < 2)
    {
        // warp 0 the gradients' running sums, warp 1 the hessians'
        double sum = 0.0;
        for (uint32_t b0 = 0; b0 < n_cut; b0 += 32)
        {
            uint32_t const b    = b0 + lane;
            float const    v    = b < n_cut ? (w == 0 ? cell[b].x : cell[b].y) : 0.0F;
            double const   mine = warp_serial_sum(v, sum);
            if (b < n_cut)
            {
                (w == 0 ? pref[b].x : pref[b].y) = mine;
            }
        }
    }
    float const  mg      = cell[nb - 1].x;
    float const  mh      = cell[nb - 1].y;
    double const node_sc = split_score(nd.sum_g, nd.sum_h, l1, l2);
    // float fields subtract in float, then widen (src/split.cpp:117-118)
    double const real_g     = static_cast<double>(nd.sum_g - mg);
    double const real_h     = static_cast<double>(nd.sum_h - mh);
    bool const   miss_empty = mg == 0.0F && mh == 0.0F;
    __syncthreads();
    uint32_t const f        = sel[j];
    int const      mc       = (mono != nullptr && f < n_mono) ? mono[f] : 0;
    uint32_t const n_dir    = miss_empty ? 1 : 2;
    double         best     = 0.0;
    uint32_t       order    = 0xFFFFFFFFu;
    double const   min_gain = tp.min_gain_to_split;
    for (uint32_t b = tid; b < n_cut; b += k_find_thr)
    {
        double2 const p = pref[b];
        for (uint32_t d = 0; d < n_dir; ++d)
        {
            double gain = 0.0;
            if (candidate_gain<float>(p.x, p.y, mg, mh, real_g, real_h, d == 0, node_sc, tp,
                                      mc, nd.lo, nd.hi, gain) &&
                gain > best && gain >= min_gain)
            {
                best  = gain;
                order = (b * 2) + d;
            }
        }
    }
    warp_best(best, order);
    if (lane == 0)
    {
        bg_s[w] = best;
        bo_s[w] = order;
    }
    __syncthreads();
    if (tid == 0)
    {
        for (uint32_t x = 1; x < k_find_thr / 32; ++x)
        {
            if (bg_s[x] > best || (bg_s[x] == best && bo_s[x] < order))
            {
                best  = bg_s[x];
                order = bo_s[x];
            }
        }
        if (order != 0xFFFFFFFFu)
        {
            out.gain  = best;
            out.bin   = order >> 1;
            out.dl    = (order & 1) == 0 ? 1 : 0;
            out.valid = 1;
        }
        cand[(i * n_sel) + j] = out;
    }
}


// ---- the quantised form's find: a warp per (node, feature) ----
//
// The cells go by in groups of 256, loaded coalesced (all in flight) and handed
// over through shared memory so that a lane holds eight consecutive bins: the
// exact integer prefix is eight adds and one warp scan, in whole cells (a
// packed cell's two sums add as one 64-bit word). Every bin's candidates are
// scored, and (largest gain, lowest bin x 2 + direction) over the warp is the
// choice of the per-(node, feature) CTA above.
//
// What bounds it is instructions: a candidate's rule in FP64, two divisions
// among it, is about 100 of them. So the children's scores are first
// approximated in float from the exact integer sums (four conversions, a
// reciprocal and a few products), and only candidates whose approximation comes
// within 2^-14 of the warp's largest take the rule: where the approximation is
// off by less than 2^-15, the true maximum and all its ties are among them, and
// their gains are the serial scan's, bit for bit. Its steps are off by 2^-20
// together, but for t = |g| - l1, which may cancel. So l1 is taken 2^-20 of itself
// too small, which makes t at least its true value less 2^-22 of it and at most
// e = 2^-19 l1 more, and a score s, the sum of t^2 / h over both children, at
// most 2 e sqrt(2 / (the least h)) sqrt(s) too large: what the largest score may
// have too much is taken off before it is compared (QNode::slack). The rule's own
// sums are right to E = 2^-49 M, M = l1 + (largest code x rows) a bound of them
// all, which changes s by 2 x + x^2 of itself, x = E sqrt(2 / (the least h) / s):
// x is at most 2^-17 where s is at least 2^-63 M^2 / (the least h), and the screen
// decides only where the warp's largest score is (QNode::floor, with a factor of
// 4 to spare). A bin without rows is skipped: its candidates are the bin before's
// over again, later in the scan's order. (Over 2,000 features: the root's find
// 15.3 to 10.5 us under ncu, 1,834 to 1,209 instructions a warp; both children of
// a pop 27 to 15.6 us. |g| - l1 in FP64 instead: 2-3% of a round; the rule for
// every candidate where l1 is not 0: 7-20% of such a round.)

constexpr uint32_t k_qfind_warps = 8;
constexpr uint32_t k_qfind_group = 8; // cells held per lane

// A cell or a sum of cells: packed in one word, or two words.
template <bool CW2> struct QCell;
template <> struct QCell<false>
{
    unsigned long long w;
    __device__ __forceinline__ void load(unsigned long long const *h, uint64_t x)
    {
        w = h[x];
    }
    __device__ __forceinline__ void store(unsigned long long *h, uint64_t x) const
    {
        h[x] = w;
    }
    __device__ __forceinline__ void clear()
    {
        w = 0;
    }
    __device__ __forceinline__ void add(QCell const &o)
    {
        w += o.w;
    }
    __device__ __forceinline__ void sub(QCell const &o)
    {
        w -= o.w;
    }
    __device__ __forceinline__ bool same(QCell const &o) const
    {
        return w == o.w;
    }
    __device__ __forceinline__ QCell up(uint32_t o) const
    {
        return {__shfl_up_sync(0xFFFFFFFFu, w, o)};
    }
    __device__ __forceinline__ QCell from(uint32_t lane) const
    {
        return {__shfl_sync(0xFFFFFFFFu, w, lane)};
    }
    __device__ __forceinline__ int64_t g() const
    {
        return static_cast<int32_t>(static_cast<uint32_t>(w >> 32));
    }
    __device__ __forceinline__ int64_t h() const
    {
        return static_cast<uint32_t>(w);
    }
};
template <> struct QCell<true>
{
    unsigned long long a, b;
    __device__ __forceinline__ void load(unsigned long long const *h, uint64_t x)
    {
        a = h[2 * x];
        b = h[(2 * x) + 1];
    }
    __device__ __forceinline__ void store(unsigned long long *h, uint64_t x) const
    {
        h[2 * x]       = a;
        h[(2 * x) + 1] = b;
    }
    __device__ __forceinline__ void clear()
    {
        a = 0;
        b = 0;
    }
    __device__ __forceinline__ void add(QCell const &o)
    {
        a += o.a;
        b += o.b;
    }
    __device__ __forceinline__ void sub(QCell const &o)
    {
        a -= o.a;
        b -= o.b;
    }
    __device__ __forceinline__ bool same(QCell const &o) const
    {
        return a == o.a && b == o.b;
    }
    __device__ __forceinline__ QCell up(uint32_t o) const
    {
        return {__shfl_up_sync(0xFFFFFFFFu, a, o), __shfl_up_sync(0xFFFFFFFFu, b, o)};
    }
    __device__ __forceinline__ QCell from(uint32_t lane) const
    {
        return {__shfl_sync(0xFFFFFFFFu, a, lane), __shfl_sync(0xFFFFFFFFu, b, lane)};
    }
    __device__ __forceinline__ int64_t g() const
    {
        return static_cast<int64_t>(a);
    }
    __device__ __forceinline__ int64_t h() const
    {
        return static_cast<int64_t>(b);
    }
};

// What the candidates of one (node, feature) share: the rule's terms, and
// those of the approximation, in units of the quantisation scales.
struct QNode
{
    double   mg, mh, node_sc, real_g, real_h, lo, hi;
    int64_t  img, irg, irh; // the missing bin's g; g and h without it
    float    fmh, l1, l2, sure, maybe;
    float    slack, floor; // of the largest score's root, and the least one that decides
    uint32_t n_dir;
    int      mc;

    // qmax: the largest code
    __device__ __forceinline__ void start(int64_t qg, int64_t qh, int64_t mqg, int64_t mqh,
                                          Node const &nd, int mono, double2 const &sc,
                                          TreeParams const &tp, float qmax)
    {
        mg      = static_cast<double>(mqg) * sc.x;
        mh      = static_cast<double>(mqh) * sc.y;
        node_sc = split_score(static_cast<double>(qg) * sc.x, static_cast<double>(qh) * sc.y,
                              tp.lambda_l1, tp.lambda_l2);
        real_g  = static_cast<double>(qg - mqg) * sc.x;
        real_h  = static_cast<double>(qh - mqh) * sc.y;
        n_dir   = (mqg == 0 && mqh == 0) ? 1 : 2;
        lo      = nd.lo;
        hi      = nd.hi;
        mc      = mono;
        img     = mqg;
        irg     = qg - mqg;
        irh     = qh - mqh;
        fmh     = static_cast<float>(mqh);
        // (an inf or NaN here makes every candidate take the rule)
        float const sx = 1.0F / static_cast<float>(sc.x);
        float const sy = 1.0F / static_cast<float>(sc.y);
        l1             = tp.lambda_l1 * sx * (1.0F - 0x1p-20F);
        l2             = tp.lambda_l2 * sy;
        // min_child_hess, which the rule compares in FP64, from both sides
        sure  = tp.min_child_hess * sy * (1.0F + 0x1p-18F);
        maybe = tp.min_child_hess * sy * (1.0F - 0x1p-18F);
        // (where nothing else keeps h off 0 it is a whole number, or the score is
        // not finite)
        float const least = fmaxf(maybe, 0.0F) + l2;
        float const q     = sqrtf(2.0F / (least > 0.0F ? least : 1.0F));
        float const m     = 0x1p-31F * q * (l1 + (qmax * static_cast<float>(nd.gcount)));
        floor             = fmaxf(1e-30F, m * m);
        slack             = 0x1p-18F * q * l1;
    }
};

// The shared memory of a warp's hand-over: a cell of padding after every
// eight, so that lanes reading their eight in step hit different banks.
template <bool CW2> struct QHand
{
    QCell<CW2> c[(32 * k_qfind_group) + 32];
    __device__ __forceinline__ static uint32_t at(uint32_t b)
    {
        return b + (b >> 3);
    }
};

// A group's cells (chunk q's bin 32 q + lane) as this lane's eight
// consecutive bins' inclusive prefixes, continued from and into carry; before
// is the prefix ahead of the first.
template <bool CW2>
__device__ __forceinline__ void qscan_group(QCell<CW2> (&v)[k_qfind_group], QHand<CW2> &hand,
                                            QCell<CW2> &carry, QCell<CW2> &before)
{
    static_assert(k_qfind_group == 8, "a lane's bins and the padding go by eights");
    uint32_t const lane = threadIdx.x & 31;
    __syncwarp(); // the last group's readers are done
#pragma unroll
    for (uint32_t q = 0; q < 8; ++q)
    {
        hand.c[QHand<CW2>::at((q * 32) + lane)] = v[q];
    }
    __syncwarp();
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i)
    {
        v[i] = hand.c[QHand<CW2>::at((lane * 8) + i)];
        if (i > 0)
        {
            v[i].add(v[i - 1]);
        }
    }
    QCell<CW2> run = v[7];
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1)
    {
        QCell<CW2> const u = run.up(o);
        if (lane >= o)
        {
            run.add(u);
        }
    }
    QCell<CW2> const total = run.from(31);
    run.sub(v[7]);
    run.add(carry);
    before = run;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i)
    {
        v[i].add(run);
    }
    carry.add(total);
}

__device__ __forceinline__ float fast_rcp(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// A group's candidates into this lane's best: bins c0 + 8 lane + i.
template <bool CW2>
__device__ __forceinline__ void qscore_group(QCell<CW2> const (&v)[k_qfind_group],
                                             QCell<CW2> const &before, uint32_t c0,
                                             uint32_t n_cut, QNode const &n, double2 const &sc,
                                             TreeParams const &tp, double &best, uint32_t &order)
{
    using Int            = std::conditional_t<CW2, int64_t, int32_t>;
    uint32_t const lane  = threadIdx.x & 31;
    uint32_t const first = c0 + (lane * 8);
    auto const     score = [&](Int g, float h) // h with l2 added
    {
        float const t = fmaxf(fabsf(static_cast<float>(g)) - n.l1, 0.0F);
        return (t * t) * fast_rcp(h);
    };
    float    about[2][8];
    float    top   = -1.0F;
    uint32_t some  = 0; // candidates of bins with rows, in scan order
    auto     prev  = before;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i)
    {
        Int const   g  = static_cast<Int>(v[i].g());
        Int const   rg = static_cast<Int>(n.irg) - g;
        float const h  = static_cast<float>(v[i].h());
        float const rh = static_cast<float>(n.irh - v[i].h());
        Int const   mg = static_cast<Int>(n.img);
        bool const  in = first + i < n_cut && (!v[i].same(prev) || first + i == 0);
        prev           = v[i];
        // missing to the left, then (where there is any) to the right
#pragma unroll
        for (uint32_t d = 0; d < 2; ++d)
        {
            about[d][i] = -1.0F;
            if (d == 1 && n.n_dir == 1) // uniform
            {
                continue;
            }
            float const hL = d == 0 ? h + n.fmh : h;
            float const hR = d == 0 ? rh : rh + n.fmh;
            float const s  = score(d == 0 ? g + mg : g, hL + n.l2) +
                            score(d == 0 ? rg : rg + mg, hR + n.l2);
            float const least = fminf(hL, hR);
            if (in && !(least < n.maybe))
            {
                about[d][i] = s;
                some |= 1u << ((2 * i) + d);
                top = least >= n.sure ? fmaxf(top, s) : top;
            }
        }
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
    }
    top = top - (n.slack * sqrtf(fmaxf(top, 0.0F)));
    // monotone candidates are chosen among by their leaf weights too, and
    // scores past the normal float range say nothing about the order: the
    // rule for them all
    float const bar = n.mc != 0 || !(top < 1e37F && top > n.floor && n.l2 < 1e30F && n.l1 < 1e30F)
                          ? -0.5F
                          : top * (1.0F - 0x1p-14F);
    uint32_t todo = 0;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i)
    {
#pragma unroll
        for (uint32_t d = 0; d < 2; ++d)
        {
            todo |= about[d][i] < bar ? 0u : 1u << ((2 * i) + d); // (NaN too)
        }
    }
    todo = bar < 0.0F ? some : todo & some;
#pragma unroll 1
    while (__any_sync(0xFFFFFFFFu, todo != 0))
    {
        if (todo != 0)
        {
            uint32_t const at = __ffs(todo) - 1;
            todo &= todo - 1;
            QCell<CW2> c = v[0];
#pragma unroll
            for (uint32_t i = 1; i < 8; ++i)
            {
                if ((at >> 1) == i)
                {
                    c = v[i];
                }
            }
            double gain = 0.0;
            if (candidate_gain<double>(static_cast<double>(c.g()) * sc.x,
                                       static_cast<double>(c.h()) * sc.y, n.mg, n.mh, n.real_g,
                                       n.real_h, (at & 1) == 0, n.node_sc, tp, n.mc, n.lo, n.hi,
                                       gain) &&
                gain > best && gain >= tp.min_gain_to_split)
            {
                best  = gain;
                order = ((first + (at >> 1)) * 2) + (at & 1);
            }
        }
    }
}

// Cuts n row segments (n <= NT) into chunks of `rows` rows with the
// whole block: segment i owns chunks [range[i], range[i + 1]), and
// seg(i, start, count, aux) describes it. One thread per segment stages its
// chunk origin and description in shared memory first (range and what seg
// reads are in global memory, written before a barrier), so a chunk's binary
// search and lookup read no global memory.
template <uint32_t NT, typename Seg>
__device__ __forceinline__ void fill_chunk_table(uint32_t n, uint32_t const *range,
                                                 uint32_t total, uint32_t rows, Seg seg,
                                                 Chunk *out)
{
    __shared__ uint32_t range_s[NT];
    __shared__ uint32_t start_s[NT];
    __shared__ uint32_t count_s[NT];
    __shared__ uint32_t aux_s[NT];
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x)
    {
        uint32_t st  = 0;
        uint32_t cnt = 0;
        uint32_t aux = 0;
        seg(i, st, cnt, aux);
        range_s[i] = range[i];
        start_s[i] = st;
        count_s[i] = cnt;
        aux_s[i]   = aux;
    }
    __syncthreads();
    for (uint32_t c = threadIdx.x; c < total; c += blockDim.x)
    {
        uint32_t lo = 0;
        uint32_t hi = n;
        while (hi - lo > 1)
        {
            uint32_t const mid = (lo + hi) >> 1;
            if (range_s[mid] <= c)
            {
                lo = mid;
            }
            else
            {
                hi = mid;
            }
        }
        uint32_t const b = (c - range_s[lo]) * rows;
        out[c]           = {lo, start_s[lo] + b, min(rows, count_s[lo] - b), aux_s[lo]};
    }
}

struct PlanArgs
{
    uint32_t const *sel;
    float const    *cuts;
    uint32_t const *cut_off;
    TreeParams      tp;
    TreeOut         t;
    Chunk          *pchunks;
    uint32_t       *pcr;
    double2        *nbound;
    HeapOut         ho;
    uint32_t       *nleft;
    uint32_t       *nright;
    uint4          *route; // per node: its split's feature, last bin, bin, direction
};

// The frontier's splits and leaves written into the tree, and the partition's
// chunk table, from every node's best split (one block of NT threads, a thread
// per node).
template <uint32_t NT>
__device__ __forceinline__ void plan_level(Ctl *ctl, Node *nodes, Best const *best, uint32_t n_cur,
                                           PlanArgs const &A)
{
    TreeParams const      tp      = A.tp;
    TreeOut const        &t       = A.t;
    HeapOut const        &ho      = A.ho;
    uint32_t const *const cut_off = A.cut_off;
    uint32_t *const       pcr     = A.pcr;
    uint32_t const i     = threadIdx.x;
    bool const     live  = i < n_cur;
    Best const     bs    = live ? best[i] : Best{};
    bool const     split = live && bs.valid != 0;
    uint32_t       n_split_total = 0;
    uint32_t const rank  = block_excl_scan<NT>(split ? 1 : 0, &n_split_total);
    uint32_t const n_nodes0 = ctl->n_nodes;
    Node           nd       = live ? nodes[i] : Node{};
    if (live)
    {
        A.nleft[i]      = 0; // the one-pass partition's per-node counters
        A.nright[i]     = 0;
        A.nbound[nd.id] = make_double2(nd.lo, nd.hi); // for a later leaf renewal
        if (split)
        {
            uint32_t const f     = A.sel[bs.feature];
            uint32_t const left  = n_nodes0 + (2 * rank);
            uint32_t const right = left + 1;
            t.feature[nd.id]      = f;
            t.value[nd.id]        = A.cuts[cut_off[f] + bs.bin];
            t.left[nd.id]         = left;
            t.right[nd.id]        = right;
            t.default_left[nd.id] = static_cast<uint8_t>(bs.dl);
            t.gain[nd.id]         = static_cast<float>(bs.gain);
            t.split_bin[nd.id]    = bs.bin;
            write_leaf_node(t, left, 0.0F);
            write_leaf_node(t, right, 0.0F);
            t.gain[left]   = 0.0F;
            t.gain[right]  = 0.0F;
            t.cover[left]  = 0.0F;
            t.cover[right] = 0.0F;
            // a demoted split's children keep these: nothing comes after to
            // write their bounds, and leaf_fix reads every leaf's
            A.nbound[left]  = make_double2(-INFINITY, INFINITY);
            A.nbound[right] = make_double2(-INFINITY, INFINITY);
            nd.flags            = 1;
            uint32_t const last = cut_off[f + 1] - cut_off[f] - 1;
            A.route[i]          = make_uint4(f, last, bs.bin, bs.dl);
            if (ho.heap != nullptr && nd.heap < k_heap_slots)
            {
                ho.heap[nd.heap] = heap_entry(f, ho.per, bs.bin, last, bs.dl != 0);
            }
        }
        else
        {
            heap_leaf(ho, nd.heap, nd.id);
            write_leaf_node(t, nd.id, leaf_value(nd, tp));
            nd.flags = 0;
        }
        nodes[i] = nd;
    }
    // partition chunk table over every frontier node
    uint32_t const nch    = live ? (nd.count + k_part_rows - 1) / k_part_rows : 0;
    uint32_t       total  = 0;
    uint32_t const c0     = block_excl_scan<NT>(nch, &total);
    if (live)
    {
        pcr[i] = c0;
    }
    if (i == 0)
    {
        pcr[n_cur]      = total;
        ctl->n_pchunks  = total;
        ctl->n_psplit   = n_split_total;
        ctl->n_nodes    = n_nodes0 + (2 * n_split_total);
        ctl->n_leaves  += n_cur - n_split_total;
    }
    __syncthreads();
    fill_chunk_table<NT>(
        n_cur, pcr, total, k_part_rows,
        [&](uint32_t x, uint32_t &st, uint32_t &cnt, uint32_t &aux)
        {
            Node const nx = nodes[x];
            st            = nx.start;
            cnt           = nx.count;
            aux           = 0;
        },
        A.pchunks);
}

// The quantised form's node totals: exact integer sums of the first selected
// feature's cells with one warp (order-free), every lane holding them.
__device__ __forceinline__ void warp_qtotals(unsigned long long const *cells, uint32_t nb,
                                             uint32_t cw, int64_t &g, int64_t &h)
{
    int64_t sg = 0;
    int64_t sh = 0;
    for (uint32_t b = threadIdx.x & 31; b < nb; b += 32)
    {
        int64_t cg, ch;
        qcell(cells, b, cw, cg, ch);
        sg += cg;
        sh += ch;
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        sg += __shfl_xor_sync(0xFFFFFFFFu, sg, o);
        sh += __shfl_xor_sync(0xFFFFFFFFu, sh, o);
    }
    g = sg;
    h = sh;
}

// The level chain: for a walked tree with packed cells and a split per node,
// the find also subtracts the larger children (parent - smaller, exact
// integers) while it reads them, a node's last block picks its split and takes
// its left totals off the split's cells, and the find's last block plans the
// partition, so that a level is the build, this, the partition and the next
// frontier's plan: four launches for six, and one pass less over the cells.
// With the tree opened beside its quantisation and the leaves renewed by the
// walk's last block, a round of depth 6 x 28 features is 33 launches for 45: us
// at 1,000 / 20,000 / 200,000 rows 233 / 249 / 250 before, 228 / 241 / 244 now,
// 64 fits in flight 235 ms for 100 rounds before, 221 now. What was measured and
// left: the partition's last block planning the next frontier (registers: the
// partition 24 to 32 us at 10,000,000 rows); two-word cells (500,000 rows 328 to
// 334) and the levelwise find (its few blocks subtract slowly: 525 to 535).
struct FindChain
{
    Ctl                      *ctl;
    Node                     *nodes;
    Best                     *best;
    int64_t                  *ltot;    // per node: (G, H) left of its split
    uint32_t                 *ticket;  // [0] the launch's, [1 + i] node i's
    unsigned long long       *hist;    // this level's cells
    unsigned long long const *parents; // the level above's; null at the root
    uint32_t const           *bpair;
    PlanArgs                  plan;
};

// (G, H) of the rows that a split sends left, off the node's cells of the
// split feature (a warp; lane 0 writes them).
__device__ __forceinline__ void left_totals(unsigned long long const *cells, uint32_t nb,
                                            uint32_t cw, Best const &bs, int64_t *out)
{
    int64_t sg = 0;
    int64_t sh = 0;
    for (uint32_t b = threadIdx.x & 31; b < nb; b += 32)
    {
        if (b <= bs.bin || (b == nb - 1 && bs.dl != 0))
        {
            int64_t cg, ch;
            qcell(cells, b, cw, cg, ch);
            sg += cg;
            sh += ch;
        }
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        sg += __shfl_xor_sync(0xFFFFFFFFu, sg, o);
        sh += __shfl_xor_sync(0xFFFFFFFFu, sh, o);
    }
    if ((threadIdx.x & 31) == 0)
    {
        out[0] = sg;
        out[1] = sh;
    }
}

// The first feature (ascending) with the largest gain among a node's
// candidates (a warp; every lane returns it).
__device__ __forceinline__ Best best_candidate(Best const *cand, uint32_t n_sel)
{
    double   g = 0.0;
    uint32_t o = 0xFFFFFFFFu;
    for (uint32_t j = threadIdx.x & 31; j < n_sel; j += 32)
    {
        Best const c = cand[j];
        if (c.valid != 0 && (c.gain > g || (c.gain == g && j < o)))
        {
            g = c.gain;
            o = j;
        }
    }
    warp_best(g, o);
    o = __shfl_sync(0xFFFFFFFFu, o, 0);
    return o == 0xFFFFFFFFu ? Best{0.0, 0, 0, 1, 0} : cand[o];
}

template <bool CW2, bool CHAIN>
__global__ void __launch_bounds__(k_qfind_warps * 32, CW2 ? 1 : 3)
    qfind_warp_kernel(Ctl const *ctl, Node const *nodes, void const *hist_v,
                      uint32_t total_cells, uint32_t const *cell_off, uint32_t const *sel_nb,
                      uint32_t const *sel, uint32_t n_sel, int8_t const *mono, uint32_t n_mono,
                      TreeParams tp, Best *cand, double2 const *qscale, uint64_t const *fgroups,
                      FindChain C)
{
    pdl_enter();
    constexpr uint32_t cw    = CW2 ? 2 : 1;
    uint32_t const     i     = blockIdx.x;
    uint32_t const     n_cur = ctl->n_cur;
    if (i >= n_cur && (!CHAIN || n_cur != 0 || i + blockIdx.y != 0))
    {
        return; // (an empty frontier is planned by the first block)
    }
    uint32_t const lane = threadIdx.x & 31;
    uint32_t const j    = (blockIdx.y * k_qfind_warps) + (threadIdx.x >> 5);
    if (i < n_cur && j < n_sel)
    {
        Node           nd   = nodes[i];
        uint32_t const nb   = sel_nb[j];
        uint32_t const f    = sel[j];
        uint32_t const off  = cell_off[j];
        auto const    *base = static_cast<unsigned long long const *>(hist_v);
        auto const *src = base + (((static_cast<uint64_t>(i) * total_cells) + off) * cw);
        // the larger child's cells: its parent's less its sibling's
        bool                      large = false;
        unsigned long long const *par   = nullptr;
        unsigned long long const *sib   = nullptr;
        if constexpr (CHAIN)
        {
            if (C.parents != nullptr)
            {
                uint32_t const *pair = C.bpair + (3 * (i >> 1));
                large                = pair[2] == i;
                par = C.parents + (((static_cast<uint64_t>(pair[0]) * total_cells) + off) * cw);
                sib = base + (((static_cast<uint64_t>(pair[1]) * total_cells) + off) * cw);
            }
            else
            {
                warp_qtotals(src, nb, cw, nd.qg, nd.qh); // the root: every row is in one cell
            }
        }
        auto const cell = [&](uint32_t b, bool keep)
        {
            QCell<CW2> c;
            if (CHAIN && large)
            {
                QCell<CW2> o;
                c.load(par, b);
                o.load(sib, b);
                c.sub(o);
                if (keep)
                {
                    c.store(C.hist + (((static_cast<uint64_t>(i) * total_cells) + off) * cw), b);
                }
            }
            else
            {
                c.load(src, b);
            }
            return c;
        };
        Best       out     = {0.0, j, 0, 1, 0};
        bool const open    = nd.gcount >= 2 * tp.min_data_in_leaf && nb >= 2;
        bool const allowed = open && interaction_allows(nd, fgroups, f);
        if (allowed)
        {
            uint32_t const   n_cut = nb - 2;
            double2 const    sc    = *qscale;
            QCell<CW2> const miss  = cell(nb - 1, lane == 0);
            if (CHAIN && large && lane == 0)
            {
                cell(nb - 2, true);
            }
            QNode n;
            n.start(nd.qg, nd.qh, miss.g(), miss.h(), nd,
                    (mono != nullptr && f < n_mono) ? mono[f] : 0, sc, tp,
                    CW2 ? 32767.0F : 127.0F);
            __shared__ QHand<CW2> hand_s[k_qfind_warps];
            QHand<CW2>           &hand  = hand_s[threadIdx.x >> 5];
            double                best  = 0.0;
            uint32_t              order = 0xFFFFFFFFu;
            QCell<CW2>            carry, before;
            carry.clear();
            for (uint32_t c0 = 0; c0 < n_cut; c0 += 32 * k_qfind_group)
            {
                QCell<CW2> v[k_qfind_group];
#pragma unroll
                for (uint32_t q = 0; q < k_qfind_group; ++q)
                {
                    uint32_t const b = c0 + (q * 32) + lane;
                    v[q].clear();
                    if (b < n_cut)
                    {
                        v[q] = cell(b, true);
                    }
                }
                qscan_group<CW2>(v, hand, carry, before);
                qscore_group<CW2>(v, before, c0, n_cut, n, sc, tp, best, order);
            }
            warp_best(best, order);
            if (order != 0xFFFFFFFFu)
            {
                out.gain  = best;
                out.bin   = order >> 1;
                out.dl    = (order & 1) == 0 ? 1 : 0;
                out.valid = 1;
            }
        }
        else if (CHAIN && large && open)
        {
            // (a constrained feature's cells: the children may ask for them)
            for (uint32_t b = lane; b < nb; b += 32)
            {
                cell(b, true);
            }
        }
        if (lane == 0)
        {
            cand[(i * n_sel) + j] = out;
        }
    }
    if constexpr (CHAIN)
    {
        if (i < n_cur)
        {
            if (!last_block(C.ticket + 1 + i, gridDim.y))
            {
                return;
            }
            if (threadIdx.x < 32)
            {
                auto const *cells = C.hist + (static_cast<uint64_t>(i) * total_cells * cw);
                Best const  bs    = best_candidate(cand + (static_cast<uint64_t>(i) * n_sel), n_sel);
                if (lane == 0)
                {
                    C.best[i] = bs;
                }
                if (bs.valid != 0)
                {
                    left_totals(cells + (static_cast<uint64_t>(cell_off[bs.feature]) * cw),
                                sel_nb[bs.feature], cw, bs, C.ltot + (2 * i));
                }
                if (C.parents == nullptr)
                {
                    int64_t g, h;
                    warp_qtotals(cells, sel_nb[0], cw, g, h);
                    if (lane == 0)
                    {
                        C.nodes[0].qg = g;
                        C.nodes[0].qh = h;
                    }
                }
            }
            if (!last_block(C.ticket, n_cur))
            {
                return;
            }
        }
        plan_level<k_qfind_warps * 32>(C.ctl, C.nodes, C.best, n_cur, C.plan);
    }
}


// ------------------------------------------------------- level split find ----
//
// update_best_for_feature_for_level (src/split.cpp:164-235): one split for
// the whole frontier. Per feature and candidate (bin, default_left), the sum
// over the frontier's nodes, in frontier order, of each node's children
// score when both children clear min_child_hess and of its own score
// otherwise (issue #60: an infeasible node no longer vetoes the cut), minus
// the sum of the nodes' scores. grid (n_sel), k_lfind_thr threads: warps
// take the nodes of a group in parallel (prefix over the cut bins: the
// exact form's serial FP64 chain, the quantised form's exact integer scan),
// then every thread adds the group's nodes for its bins in frontier order,
// so the FP64 sums follow the reference's order bit for bit.
constexpr uint32_t k_lfind_thr = 1024;

struct LevelNode
{
    double score; // the node's own split score
    double real_g;
    double real_h;
    double mg;    // its missing cell
    double mh;
};

template <typename M>
__device__ __forceinline__ double level_term(double lg, double lh, M mg, M mh, double real_g,
                                             double real_h, bool dl, double node_score,
                                             TreeParams const &tp)
{
    double const rg = real_g - lg;
    double const rh = real_h - lh;
    double const gL = lg + (dl ? static_cast<double>(mg) : 0.0);
    double const hL = lh + (dl ? static_cast<double>(mh) : 0.0);
    double const gR = rg + (!dl ? static_cast<double>(mg) : 0.0);
    double const hR = rh + (!dl ? static_cast<double>(mh) : 0.0);
    double const mch = tp.min_child_hess;
    if (hL < mch || hR < mch)
    {
        return node_score;
    }
    double const l1 = tp.lambda_l1;
    double const l2 = tp.lambda_l2;
    return split_score(gL, hL, l1, l2) + split_score(gR, hR, l1, l2);
}

template <bool Q>
__global__ void __launch_bounds__(k_lfind_thr)
    level_find_kernel(Ctl const *ctl, Node const *nodes, void const *hist_v,
                      uint32_t total_cells, uint32_t const *cell_off, uint32_t const *sel_nb,
                      uint32_t n_sel, TreeParams tp, Best *cand, uint32_t max_nb,
                      uint32_t group, double2 const *qscale, uint32_t cw)
{
    pdl_enter();
    extern __shared__ unsigned char smem_raw[];
    __shared__ LevelNode ln_s[k_lfind_thr / 32];
    __shared__ double    bg_s[k_lfind_thr / 32];
    __shared__ uint32_t  bo_s[k_lfind_thr / 32];
    constexpr uint32_t   k_bins_per_thr = k_max_bins / k_lfind_thr;
    uint32_t const       j     = blockIdx.x;
    uint32_t const       tid   = threadIdx.x;
    uint32_t const       lane  = tid & 31;
    uint32_t const       w     = tid >> 5;
    uint32_t const       n_cur = ctl->n_cur;
    uint32_t const       nb    = sel_nb[j];
    Best                 out   = {0.0, j, 0, 1, 0};
    if (nb < 3 || n_cur == 0)
    {
        if (tid == 0)
        {
            cand[j] = out;
        }
        return;
    }
    uint32_t const n_cut = nb - 2;
    auto          *pref  = reinterpret_cast<double2 *>(smem_raw); // [group][max_nb]
    double         acc[2 * k_bins_per_thr];
#pragma unroll
    for (uint32_t x = 0; x < 2 * k_bins_per_thr; ++x)
    {
        acc[x] = 0.0;
    }
    double         parent_sum = 0.0;
    double2 const  sc         = Q ? *qscale : make_double2(1.0, 1.0);
    for (uint32_t g0 = 0; g0 < n_cur; g0 += group)
    {
        // warp w prefixes node g0 + w of the group
        if (w < group && g0 + w < n_cur)
        {
            uint32_t const p   = g0 + w;
            Node const     nd  = nodes[p];
            double2       *pr  = pref + (static_cast<uint64_t>(w) * max_nb);
            auto const    *src = static_cast<unsigned long long const *>(hist_v) +
                              (((static_cast<uint64_t>(p) * total_cells) + cell_off[j]) * cw);
            if constexpr (Q)
            {
                uint32_t const run = (n_cut + 31) / 32;
                uint32_t const b0  = min(n_cut, lane * run);
                uint32_t const b1  = min(n_cut, b0 + run);
                int64_t        tg  = 0;
                int64_t        th  = 0;
                for (uint32_t b = b0; b < b1; ++b)
                {
                    int64_t cg, ch;
                    qcell(src, b, cw, cg, ch);
                    tg += cg;
                    th += ch;
                }
                int64_t eg = tg;
                int64_t eh = th;
#pragma unroll
                for (uint32_t o = 1; o < 32; o <<= 1)
                {
                    int64_t const ug = __shfl_up_sync(0xFFFFFFFFu, eg, o);
                    int64_t const uh = __shfl_up_sync(0xFFFFFFFFu, eh, o);
                    if (lane >= o)
                    {
                        eg += ug;
                        eh += uh;
                    }
                }
                int64_t pg = eg - tg;
                int64_t ph = eh - th;
                for (uint32_t b = b0; b < b1; ++b)
                {
                    int64_t cg, ch;
                    qcell(src, b, cw, cg, ch);
                    pg += cg;
                    ph += ch;
                    pr[b] = make_double2(static_cast<double>(pg) * sc.x,
                                         static_cast<double>(ph) * sc.y);
                }
                if (lane == 0)
                {
                    int64_t mqg, mqh;
                    qcell(src, nb - 1, cw, mqg, mqh);
                    LevelNode     l;
                    l.score  = split_score(static_cast<double>(nd.qg) * sc.x,
                                           static_cast<double>(nd.qh) * sc.y, tp.lambda_l1,
                                           tp.lambda_l2);
                    l.real_g = static_cast<double>(nd.qg - mqg) * sc.x;
                    l.real_h = static_cast<double>(nd.qh - mqh) * sc.y;
                    l.mg     = static_cast<double>(mqg) * sc.x;
                    l.mh     = static_cast<double>(mqh) * sc.y;
                    ln_s[w]  = l;
                }
            }
            else
            {
                auto const *cell = reinterpret_cast<float2 const *>(src);
                // Histogram::fill_prefix (include/bonsai/histogram.hpp:139-160):
                // double running sums, each entry stored as a float cell
                double sg = 0.0;
                double sh = 0.0;
                for (uint32_t b0 = 0; b0 < n_cut; b0 += 32)
                {
                    uint32_t const b  = b0 + lane;
                    float2 const   c  = b < n_cut ? cell[b] : make_float2(0.0F, 0.0F);
                    double const   lg = warp_serial_sum(c.x, sg);
                    double const   lh = warp_serial_sum(c.y, sh);
                    if (b < n_cut)
                    {
                        pr[b] = make_double2(static_cast<float>(lg), static_cast<float>(lh));
                    }
                }
                if (lane == 0)
                {
                    float2 const m = cell[nb - 1];
                    LevelNode    l;
                    l.score  = split_score(nd.sum_g, nd.sum_h, tp.lambda_l1, tp.lambda_l2);
                    // float fields subtract in float, then widen
                    l.real_g = static_cast<double>(nd.sum_g - m.x);
                    l.real_h = static_cast<double>(nd.sum_h - m.y);
                    l.mg     = m.x;
                    l.mh     = m.y;
                    ln_s[w]  = l;
                }
            }
        }
        __syncthreads();
        uint32_t const gn = min(group, n_cur - g0);
        // every (node, bin) pair's two terms, all threads at once (the FP64
        // divisions are independent), in place of the pair's prefix
        for (uint32_t x = tid; x < gn * n_cut; x += k_lfind_thr)
        {
            uint32_t const  q    = x / n_cut;
            uint32_t const  b    = x - (q * n_cut);
            LevelNode const l    = ln_s[q];
            double2        *cell = pref + ((static_cast<uint64_t>(q) * max_nb) + b);
            double2 const   p2   = *cell;
            double          t0;
            double          t1;
            if constexpr (Q)
            {
                t0 = level_term<double>(p2.x, p2.y, l.mg, l.mh, l.real_g, l.real_h, true,
                                        l.score, tp);
                t1 = level_term<double>(p2.x, p2.y, l.mg, l.mh, l.real_g, l.real_h, false,
                                        l.score, tp);
            }
            else
            {
                float const mg = static_cast<float>(l.mg);
                float const mh = static_cast<float>(l.mh);
                t0 = level_term<float>(p2.x, p2.y, mg, mh, l.real_g, l.real_h, true, l.score,
                                       tp);
                t1 = level_term<float>(p2.x, p2.y, mg, mh, l.real_g, l.real_h, false, l.score,
                                       tp);
            }
            *cell = make_double2(t0, t1);
        }
        __syncthreads();
        // then each bin adds the group's terms in frontier order
        for (uint32_t q = 0; q < gn; ++q)
        {
            double2 const *pr = pref + (static_cast<uint64_t>(q) * max_nb);
#pragma unroll
            for (uint32_t x = 0; x < k_bins_per_thr; ++x)
            {
                uint32_t const b = tid + (x * k_lfind_thr);
                if (b < n_cut)
                {
                    double2 const t2 = pr[b];
                    acc[2 * x] += t2.x;
                    acc[(2 * x) + 1] += t2.y;
                }
            }
            parent_sum += ln_s[q].score;
        }
        __syncthreads();
    }
    // every node's missing cell empty: both routings sum the same, and the
    // first (default left) wins the strict > below, as the serial scan does
    double         best     = 0.0;
    uint32_t       order    = 0xFFFFFFFFu;
    double const   min_gain = tp.min_gain_to_split;
#pragma unroll
    for (uint32_t x = 0; x < k_bins_per_thr; ++x)
    {
        uint32_t const b = tid + (x * k_lfind_thr);
        if (b < n_cut)
        {
            for (uint32_t d = 0; d < 2; ++d)
            {
                double const gain = acc[(2 * x) + d] - parent_sum;
                if (gain > best && gain >= min_gain)
                {
                    best  = gain;
                    order = (b * 2) + d;
                }
            }
        }
    }
    warp_best(best, order);
    if (lane == 0)
    {
        bg_s[w] = best;
        bo_s[w] = order;
    }
    __syncthreads();
    if (tid == 0)
    {
        for (uint32_t x = 1; x < k_lfind_thr / 32; ++x)
        {
            if (bg_s[x] > best || (bg_s[x] == best && bo_s[x] < order))
            {
                best  = bg_s[x];
                order = bo_s[x];
            }
        }
        if (order != 0xFFFFFFFFu)
        {
            out.gain  = best;
            out.bin   = order >> 1;
            out.dl    = (order & 1) == 0 ? 1 : 0;
            out.valid = 1;
        }
        cand[j] = out;
    }
}

// ------------------------------------------------------------- planning ----

__global__ void __launch_bounds__(k_plan_thr)
    plan_kernel(Ctl *ctl, Node *nodes, Best const *cand, Best *best, uint32_t n_sel,
                bool level, PlanArgs A)
{
    pdl_enter();
    __shared__ Best    level_s;
    uint32_t const n_cur = ctl->n_cur;
    uint32_t const lane  = threadIdx.x & 31;
    uint32_t const w     = threadIdx.x >> 5;
    if (level)
    {
        // one split for the level (reduce_in_feature_order, src/split.cpp:239-250),
        // broadcast to every frontier node
        if (w == 0)
        {
            double   g = 0.0;
            uint32_t o = 0xFFFFFFFFu;
            for (uint32_t j = lane; j < n_sel; j += 32)
            {
                Best const c = cand[j];
                if (c.valid != 0 && (c.gain > g || (c.gain == g && j < o)))
                {
                    g = c.gain;
                    o = j;
                }
            }
            warp_best(g, o);
            if (lane == 0)
            {
                level_s = o == 0xFFFFFFFFu ? Best{0.0, 0, 0, 1, 0} : cand[o];
            }
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < n_cur; i += k_plan_thr)
        {
            best[i] = level_s;
        }
    }
    // per node: the first feature (ascending) holding the largest gain
    for (uint32_t i = w; !level && i < n_cur; i += k_plan_thr / 32)
    {
        double   g = 0.0;
        uint32_t o = 0xFFFFFFFFu;
        for (uint32_t j = lane; j < n_sel; j += 32)
        {
            Best const c = cand[(i * n_sel) + j];
            if (c.valid != 0 && (c.gain > g || (c.gain == g && j < o)))
            {
                g = c.gain;
                o = j;
            }
        }
        warp_best(g, o);
        if (lane == 0)
        {
            best[i] = o == 0xFFFFFFFFu ? Best{0.0, 0, 0, 1, 0} : cand[(i * n_sel) + o];
        }
    }
    __syncthreads();
    plan_level<k_plan_thr>(ctl, nodes, best, n_cur, A);
}

// ----------------------------------------------------------------- leafwise ----
//
// One heap pop of the leafwise grower (LeafwiseGrower::grow,
// src/grower_impl.hpp:744-850; split_node, src/step/primitives.hpp:381-430): the
// popped node's segment is partitioned with the two partition passes (stable)
// into the same places of the other half of the row buffer, where its
// children then lie; its smaller child's histograms are built into a free
// slot of a histogram pool, the larger child is subtracted in place in the
// parent's slot (finish_split), and both children's best splits are found.

struct LeafPop
{
    Node     node; // the popped node: its segment of the row buffer, totals, bounds
    Best     best; // its split
    uint32_t left_id;
    uint32_t right_id;
    uint32_t parent_slot;
    uint32_t small_slot;
};

// A pop's results. (The flags have a line of their own: a CTA that has read
// them still sees what other CTAs of its launch write behind them.)
struct LeafOut
{
    alignas(128) uint32_t split; // 0: the partition emptied a side (the split is demoted)
    uint32_t small_left;
    alignas(128) Node child[2];
    Best best[2];
};

// After partition pass 1: the chunks' left bases, the node's left count, and
// either the demotion (a side came out empty) or the two children (in the
// other half of the row buffer), the smaller child's build chunks and the
// pool slots each child's histograms will sit in. Run by the pass's last CTA
// (a launch of its own took about 4 us of a pop).
struct LeafPlanArgs
{
    Ctl           *ctl;
    Chunk const   *pchunks;
    uint32_t      *pleft, *prbase, *nleft, *dst, *build, *brange, *bbase;
    Chunk         *bchunks;
    uint32_t      *bpair;
    Node          *nodes, *next;
    uint32_t      *slot_of;
    LeafOut       *out;
    uint32_t       crows;
    uint32_t       half; // rows of one half of the row buffer; 0: the children's rows are
                          // copied back into their parent's places
    LeafPop const *pp;
    uint32_t      *ticket;
};

// The popped node's scattered rows back into its segment (unless the
// partition emptied a side, which scatters nothing).
constexpr uint32_t k_far_rows = 0x80000000u;

__global__ void __launch_bounds__(k_threads)
    leaf_copyback_kernel(LeafPop const *pp, LeafOut const *out, uint32_t const *from, uint32_t *to)
{
    pdl_enter();
    if (out->split == 0)
    {
        return;
    }
    uint64_t const start = pp->node.start;
    uint64_t const count = pp->node.count;
    for (uint64_t i = (uint64_t{blockIdx.x} * k_threads) + threadIdx.x; i < count;
         i += uint64_t{gridDim.x} * k_threads)
    {
        to[start + i] = from[start + i];
    }
}

template <uint32_t NT> __device__ __forceinline__ void leaf_plan(LeafPlanArgs const &A)
{
    LeafPop const  p    = *A.pp;
    uint32_t const n_ch = A.ctl->n_pchunks;
    uint32_t const per  = (n_ch + NT - 1) / NT;
    uint32_t const c_a  = min(n_ch, threadIdx.x * per);
    uint32_t const c_b  = min(n_ch, c_a + per);
    uint32_t       sum  = 0;
    for (uint32_t c = c_a; c < c_b; ++c)
    {
        sum += __ldcg(&A.pleft[c]);
    }
    uint32_t       nl   = 0;
    uint32_t const base = block_excl_scan<NT>(sum, &nl);
    for (uint32_t c = c_a, run = base; c < c_b; ++c)
    {
        uint32_t const v = __ldcg(&A.pleft[c]);
        A.pleft[c]       = run;
        A.prbase[c]      = (A.pchunks[c].begin - p.node.start) - run;
        run += v;
    }
    uint32_t const count = p.node.count;
    uint32_t const nr    = count - nl;
    bool const     split = nl != 0 && nl != count;
    bool const     sl    = nl <= nr; // the left child wins a size tie
    uint32_t const sc    = sl ? nl : nr;
    uint32_t const to0   = A.half == 0                ? p.node.start
                           : p.node.start >= A.half ? p.node.start - A.half
                                                    : p.node.start + A.half;
    uint32_t const sb    = to0 + (sl ? 0 : nl);
    uint32_t const nchb  = split ? (sc + A.crows - 1) / A.crows : 0;
    if (threadIdx.x == 0)
    {
        A.nleft[0]        = nl;
        A.out->split      = split ? 1 : 0;
        A.out->small_left = sl ? 1 : 0;
        A.ctl->n_build    = split ? 1 : 0;
        A.ctl->n_bchunks  = nchb;
        A.ctl->n_splits   = split ? 1 : 0;
        A.ctl->built_rows = split ? sc : 0;
        if (!split)
        {
            A.nodes[0].flags |= 2; // the scatter leaves a demoted node's rows alone
        }
        else
        {
            A.dst[0]    = to0;
            Node L      = p.node;
            L.start     = to0;
            L.count     = nl;
            L.gcount    = nl;
            L.id        = p.left_id;
            L.flags     = 0;
            Node R      = p.node;
            R.start     = to0 + nl;
            R.count     = nr;
            R.gcount    = nr;
            R.id        = p.right_id;
            R.flags     = 0;
            A.next[0]    = L;
            A.next[1]    = R;
            A.build[0]   = p.small_slot;
            A.brange[0]  = 0;
            A.brange[1]  = nchb;
            A.bbase[0]   = 0;
            A.slot_of[0] = sl ? p.small_slot : p.parent_slot;
            A.slot_of[1] = sl ? p.parent_slot : p.small_slot;
            A.bpair[0]   = p.parent_slot;
            A.bpair[1]   = p.small_slot;
            A.bpair[2]   = p.parent_slot;
        }
    }
    for (uint32_t c = threadIdx.x; c < nchb; c += NT)
    {
        uint32_t const b = c * A.crows;
        A.bchunks[c]     = {0, sb + b, min(A.crows, sc - b), 0};
    }
}

// Partition pass 1: each warp routes a contiguous run of the chunk's rows
// (lanes = consecutive rows, coalesced), keeps the directions as a bitmask
// (one word per 32 rows) so pass 2 never re-reads the bins, and the block
// sums the left counts.
constexpr uint32_t k_warp_rows = k_part_rows / (k_threads / 32); // 512

// LEAF: one node's chunks (a leafwise pop), whose last CTA plans its children.
template <typename BinT, bool LEAF>
__global__ void __launch_bounds__(k_threads)
    pcount_kernel(Ctl const *ctl, Chunk const *pchunks, Node const *nodes,
                  Best const *best, uint32_t const *__restrict__ rows,
                  void const *__restrict__ bins, uint64_t n_pad, uint32_t const *sel,
                  uint32_t const *sel_nb, uint32_t *__restrict__ pleft,
                  uint32_t *__restrict__ dirs, LeafPlanArgs lp)
{
    pdl_enter();
    __shared__ uint32_t wsum[k_threads / 32];
    uint32_t const      c = blockIdx.x;
    if (c >= ctl->n_pchunks)
    {
        return;
    }
    Chunk const ch = pchunks[c];
    if ((nodes[ch.node].flags & 1) == 0)
    {
        if (threadIdx.x == 0)
        {
            pleft[c] = 0; // a leaf's chunk routes nothing
        }
        return;
    }
    Best const     bs   = best[ch.node];
    uint32_t const f    = sel[bs.feature];
    uint32_t const last = sel_nb[bs.feature] - 1;
    BinT const    *col  = static_cast<BinT const *>(bins) + (static_cast<uint64_t>(f) * n_pad);
    uint32_t const lane = threadIdx.x & 31;
    uint32_t const w    = threadIdx.x >> 5;
    uint32_t      *dw   = dirs + (static_cast<uint64_t>(c) * (k_part_rows / 32));
    uint32_t const k0   = (w * k_warp_rows) + lane;
    // every row id of the warp's run, then every code, then the ballots:
    // all loads in flight together
    constexpr uint32_t steps = k_warp_rows / 32;
    uint32_t           r[steps];
#pragma unroll
    for (uint32_t i = 0; i < steps; ++i)
    {
        uint32_t const k = k0 + (32 * i);
        r[i]             = k < ch.count ? rows[ch.begin + k] : k_leaf_flag;
    }
    // (plain loads: nodes splitting on the same feature share the column's
    // sectors, which an evict-first hint would give up early)
    uint32_t b[steps];
#pragma unroll
    for (uint32_t i = 0; i < steps; ++i)
    {
        b[i] = r[i] != k_leaf_flag ? static_cast<uint32_t>(col[r[i]]) : 0u;
    }
    uint32_t n = 0;
#pragma unroll
    for (uint32_t i = 0; i < steps; ++i)
    {
        bool const     lf = r[i] != k_leaf_flag && routes_left(b[i], last, bs.bin, bs.dl != 0);
        uint32_t const m  = __ballot_sync(0xFFFFFFFFu, lf);
        if (lane == i)
        {
            dw[(w * steps) + i] = m;
        }
        n += __popc(m);
    }
    if (lane == 0)
    {
        wsum[w] = n;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        uint32_t t = 0;
        for (uint32_t x = 0; x < k_threads / 32; ++x)
        {
            t += wsum[x];
        }
        pleft[c] = t;
    }
    if constexpr (LEAF)
    {
        __shared__ bool last_s;
        if (threadIdx.x == 0)
        {
            __threadfence();
            last_s = atomicAdd(lp.ticket, 1U) == ctl->n_pchunks - 1;
        }
        __syncthreads();
        if (last_s)
        {
            __threadfence();
            leaf_plan<k_threads>(lp);
            if (threadIdx.x == 0)
            {
                *lp.ticket = 0; // ready for the next pop
            }
        }
    }
}

// A sharded level's per-node left counts before they are combined across
// shards: the sum of the node's chunks' counts from partition pass 1.
__global__ void __launch_bounds__(k_plan_thr)
    node_left_kernel(Ctl const *ctl, uint32_t const *pcr, uint32_t const *pleft,
                     uint64_t *gleft, uint32_t n_slots)
{
    pdl_enter();
    uint32_t const n_cur = ctl->n_cur;
    for (uint32_t i = threadIdx.x; i < n_slots; i += k_plan_thr)
    {
        uint64_t nl = 0;
        if (i < n_cur)
        {
            for (uint32_t c = pcr[i]; c < pcr[i + 1]; ++c)
            {
                nl += pleft[c];
            }
        }
        gleft[i] = nl;
    }
}

struct Plan2Args
{
    Ctl            *ctl;
    Node           *nodes;
    Node           *next;
    Best const     *best;
    Chunk const    *pchunks;
    uint32_t const *pcr;
    uint32_t       *pleft, *prbase, *nleft, *dst, *bpair, *build, *brange;
    Chunk          *bchunks;
    TreeParams      tp;
    TreeOut         t;
    uint32_t        crows;
    uint32_t       *bbase;
    bool            level;
    uint64_t const *gleft;
    uint64_t const *fgroups;
    HeapOut         ho;
    // one-pass partition: per node, the exact sums of its left child, from
    // which both children take their totals and monotone bounds
    int64_t const  *ltot;
    uint32_t const *sel;
    int8_t const   *mono;
    uint32_t        n_mono;
    double2 const  *qscale;
    // the last level of such a tree: the children are its last leaves
    bool      last;
    double2  *nbound;
    uint32_t *tree_no;
    uint32_t  tree_step;
};

// The children's bounds after a split on a constrained feature, from their
// integer totals.
__device__ __forceinline__ void split_bounds(Node &L, Node &R, Node const &par, int mc,
                                             double2 const &sc, TreeParams const &tp)
{
    double const l1  = tp.lambda_l1;
    double const l2  = tp.lambda_l2;
    double const wl  = bounded_leaf_weight(static_cast<double>(L.qg) * sc.x,
                                           static_cast<double>(L.qh) * sc.y, l1, l2, par.lo,
                                           par.hi);
    double const wr  = bounded_leaf_weight(static_cast<double>(R.qg) * sc.x,
                                           static_cast<double>(R.qh) * sc.y, l1, l2, par.lo,
                                           par.hi);
    double const mid = 0.5 * (wl + wr);
    if (mc > 0)
    {
        L.hi = fmin(L.hi, mid);
        R.lo = fmax(R.lo, mid);
    }
    else
    {
        L.lo = fmax(L.lo, mid);
        R.hi = fmin(R.hi, mid);
    }
}

// After a level's partition: the next frontier, its smaller children's build
// chunks, and the demotion of splits that left a side empty (one block of NT
// threads, a thread per node). FUSED: the one-pass partition, which has
// counted and placed the rows already; the frontier advances here.
template <uint32_t NT, bool FUSED> __device__ __forceinline__ void plan_children(Plan2Args const &A)
{
    Ctl *const            ctl     = A.ctl;
    Node *const           nodes   = A.nodes;
    Node *const           next    = A.next;
    Chunk const *const    pchunks = A.pchunks;
    uint32_t const *const pcr     = A.pcr;
    uint32_t *const       pleft   = A.pleft;
    uint32_t *const       prbase  = A.prbase;
    uint32_t *const       nleft   = A.nleft;
    uint32_t *const       bpair   = A.bpair;
    uint32_t *const       build   = A.build;
    uint32_t *const       brange  = A.brange;
    uint32_t *const       bbase   = A.bbase;
    TreeParams const      tp      = A.tp;
    TreeOut const        &t       = A.t;
    uint32_t const        crows   = A.crows;
    bool const            level   = A.level;
    uint64_t const *const gleft   = A.gleft;
    HeapOut const        &ho      = A.ho;
    __shared__ uint32_t grand_s;
    __shared__ uint32_t flags_s[NT]; // per node: flags, start, prefix origin
    __shared__ uint32_t start_s[NT];
    __shared__ uint32_t p0_s[NT];
    uint32_t const      n_cur = ctl->n_cur;
    uint32_t const      n_ch  = ctl->n_pchunks;
    // A. exclusive prefix of the chunks' left counts over the whole level
    //    (leaf chunks count zero), each thread a contiguous run of chunks
    //    (the one-pass partition placed its rows already: no chunk runs)
    uint32_t const per = FUSED ? 0 : (n_ch + NT - 1) / NT;
    uint32_t const c_a = min(n_ch, threadIdx.x * per);
    uint32_t const c_b = min(n_ch, c_a + per);
    uint32_t       sum = 0;
    for (uint32_t c = c_a; c < c_b; ++c)
    {
        sum += pleft[c];
    }
    uint32_t       grand = 0;
    uint32_t const base  = block_excl_scan<NT>(sum, &grand);
    for (uint32_t c = c_a, run = base; c < c_b; ++c)
    {
        uint32_t const v = pleft[c];
        pleft[c]         = run;
        run += v;
    }
    if (threadIdx.x == 0)
    {
        grand_s = grand;
    }
    __syncthreads();
    // B. per split node: its left count, or demotion when a side is empty
    uint32_t const i    = threadIdx.x;
    bool const     live = i < n_cur;
    Node           nd   = live ? nodes[i] : Node{};
    bool           surv = false;
    uint32_t       nl   = 0;
    uint32_t       gnl  = 0; // rows routed left over every shard
    uint32_t       p0   = 0;
    if (live && (nd.flags & 1) != 0)
    {
        if (FUSED)
        {
            nl = nleft[i]; // the one-pass partition's left counter
        }
        else
        {
            uint32_t const c0 = pcr[i];
            uint32_t const c1 = pcr[i + 1];
            // a node without chunks (a level split of an empty node) past
            // the last chunk: its prefix origin is the grand total
            p0       = c0 < n_ch ? pleft[c0] : grand_s;
            nl       = (c1 < n_ch ? pleft[c1] : grand_s) - p0;
            nleft[i] = nl;
        }
        gnl               = gleft != nullptr ? static_cast<uint32_t>(gleft[i]) : nl;
        if (!level && (gnl == 0 || gnl == nd.gcount))
        {
            // demote_empty_splits: the parent is a leaf after all (a level
            // split applies to every node, empty children included)
            nd.flags |= 2;
            write_leaf_node(t, nd.id, leaf_value(nd, tp));
            t.gain[nd.id] = 0.0F;
            nodes[i]      = nd;
            heap_leaf(ho, nd.heap, nd.id);
        }
        else
        {
            surv = true;
        }
    }
    if (live)
    {
        flags_s[i] = nd.flags;
        start_s[i] = nd.start;
        p0_s[i]    = p0; // the node's prefix origin, consumed by C below
    }
    __syncthreads();
    // C. per chunk of a split node: its left and right write bases
    for (uint32_t c = threadIdx.x; !FUSED && c < n_ch; c += NT)
    {
        Chunk const    ch = pchunks[c];
        uint32_t const fl = flags_s[ch.node];
        if ((fl & 1) != 0 && (fl & 2) == 0)
        {
            uint32_t const lb = pleft[c] - p0_s[ch.node];
            pleft[c]          = lb;
            prbase[c]         = (ch.begin - start_s[ch.node]) - lb;
        }
    }
    __syncthreads();
    // D. survivors: their children in the next frontier, and the chunk table
    //    of the smaller children whose histograms are built
    uint32_t       n_surv     = 0;
    uint32_t const k          = block_excl_scan<NT>(surv ? 1 : 0, &n_surv);
    uint32_t       rows_total = 0;
    uint32_t const start = block_excl_scan<NT>(surv ? nd.count : 0, &rows_total);
    uint32_t small_count = 0;
    if (surv)
    {
        // the children's rows: compacted by pscatter, or where the one-pass
        // partition left them (the parent's segment, lefts first)
        uint32_t const s0   = FUSED ? nd.start : start;
        A.dst[i]            = s0;
        uint32_t const nr   = nd.count - nl;
        uint32_t const gnr  = nd.gcount - gnl;
        uint32_t const lid  = t.left[nd.id];
        uint32_t const rid  = t.right[nd.id];
        Node           L{s0, nl, lid, 0, 0.0F, 0.0F, nd.lo, nd.hi, 0, 0, gnl, 0, 0};
        Node           R{s0 + nl, nr, rid, 0, 0.0F, 0.0F, nd.lo, nd.hi, 0, 0, gnr, 0, 0};
        L.heap              = (2 * nd.heap) + 1;
        R.heap              = (2 * nd.heap) + 2;
        interaction_children(nd, A.fgroups, t.feature[nd.id], L, R);
        if (FUSED && A.ltot != nullptr)
        {
            L.qg              = A.ltot[2 * i];
            L.qh              = A.ltot[(2 * i) + 1];
            R.qg              = nd.qg - L.qg;
            R.qh              = nd.qh - L.qh;
            uint32_t const f  = A.sel[A.best[i].feature];
            int const      mc = (A.mono != nullptr && f < A.n_mono) ? A.mono[f] : 0;
            if (mc != 0)
            {
                split_bounds(L, R, nd, mc, *A.qscale, tp);
            }
        }
        if (FUSED && A.last)
        {
            A.nbound[lid] = make_double2(L.lo, L.hi);
            A.nbound[rid] = make_double2(R.lo, R.hi);
            heap_leaf(ho, L.heap, lid); // (leaves of value 0 until the walk's sums)
            heap_leaf(ho, R.heap, rid);
        }
        next[2 * k]         = L;
        next[(2 * k) + 1]   = R;
        t.cover[lid]        = static_cast<float>(gnl);
        t.cover[rid]        = static_cast<float>(gnr);
        // the smaller child over the whole fit: every shard builds the same one
        bool const left_sm  = gnl <= gnr;
        bpair[(3 * k) + 0]  = i;
        bpair[(3 * k) + 1]  = (2 * k) + (left_sm ? 0 : 1);
        bpair[(3 * k) + 2]  = (2 * k) + (left_sm ? 1 : 0);
        build[k]            = (2 * k) + (left_sm ? 0 : 1);
        small_count         = left_sm ? nl : nr;
    }
    uint32_t const nch   = surv ? (small_count + crows - 1) / crows : 0;
    uint32_t       nch_t = 0;
    uint32_t const c0    = block_excl_scan<NT>(nch, &nch_t);
    uint32_t       built = 0;
    uint32_t const pbase = block_excl_scan<NT>(small_count, &built);
    if (surv)
    {
        brange[k] = c0;
        bbase[k]  = pbase; // the built node's payload base
    }
    uint32_t n_dem = 0;
    block_excl_scan<NT>((live && (nd.flags & 2) != 0) ? 1 : 0, &n_dem);
    if (i == 0)
    {
        brange[n_surv]  = nch_t;
        ctl->n_leaves  += n_dem;
        ctl->n_next     = 2 * n_surv;
        if (FUSED && A.ltot != nullptr)
        {
            ctl->n_cur = 2 * n_surv;
        }
        ctl->n_splits   = n_surv;
        ctl->n_build    = n_surv;
        ctl->n_bchunks  = nch_t;
        ctl->built_rows = built;
        if (n_surv > 0)
        {
            ctl->depth += 1;
        }
        if (FUSED && A.last)
        {
            t.meta[0]   = ctl->n_nodes;
            t.meta[1]   = ctl->depth;
            t.meta[2]   = ctl->n_leaves + (2 * n_surv);
            *A.tree_no += A.tree_step; // (the tree's roundings are done)
        }
    }
    if (FUSED && A.last)
    {
        return;
    }
    __syncthreads();
    fill_chunk_table<NT>(
        n_surv, brange, nch_t, crows,
        [&](uint32_t x, uint32_t &st, uint32_t &cnt, uint32_t &aux)
        {
            Node const sm = next[build[x]];
            st            = sm.start;
            cnt           = sm.count;
            aux           = bbase[x];
        },
        A.bchunks);
}

template <bool FUSED> __global__ void __launch_bounds__(k_plan_thr) plan2_kernel(Plan2Args A)
{
    pdl_enter();
    plan_children<k_plan_thr, FUSED>(A);
}

// Rows of this level's leaves (never split, or demoted): their leaf id and
// the fused score update scores[r] += lr * value.
__global__ void __launch_bounds__(k_threads)
    stamp_kernel(Ctl const *ctl, Chunk const *pchunks, Node const *nodes,
                 uint32_t const *rows, TreeOut t, uint32_t *leaf_id, float *scores,
                 float lr)
{
    pdl_enter();
    uint32_t const c = blockIdx.x;
    if (c >= ctl->n_pchunks)
    {
        return;
    }
    Chunk const ch = pchunks[c];
    Node const  nd = nodes[ch.node];
    if ((nd.flags & 1) != 0 && (nd.flags & 2) == 0)
    {
        return;
    }
    float const v = t.value[nd.id];
    for (uint32_t k = threadIdx.x; k < ch.count; k += k_threads)
    {
        uint32_t const r = rows[ch.begin + k];
        if (leaf_id != nullptr)
        {
            leaf_id[r] = nd.id;
        }
        if (scores != nullptr)
        {
            scores[r] = scores[r] + (lr * v);
        }
    }
}

// The final walk, for trees grown over every row: each row (one thread,
// rows in order) walks the finished tree through its 32-byte mirror tiles
// with the partition's own rule (routes_left on the split bin, the last bin
// following default_left), so it reaches the leaf whose segment held it --
// and rows read in order are coalesced, where the partitioned rows are a
// gather. The walk takes a fixed number of steps through the tree's
// decision heap (a leaf above the last level repeats down its left spine, and
// the last level's slot names the leaf). One pass (exact form) updates
// scores[r] = scores[r] + lr * value -- the stamp's arithmetic -- and the
// leaf ids and, for a resident booster, writes the next round's gradient
// pairs and their maxima. The quantised form renews its leaves from
// full-precision gradients first: pass A walks and sums each leaf's
// (g, h) as exact fixed-point integers (u / max |g| and u / max h per unit,
// u = 2^38 up to 2^24 rows and halved per doubling above, so no sum passes
// 2^62; integer sums are order-free, hence deterministic), a one-CTA kernel
// turns them into FP64 Newton values, and
// pass B applies them from the leaf id pass A recorded.
constexpr uint32_t k_walk_nodes = 512;     // a depth-8 tree has at most 511

struct WalkArgs
{
    float        *scores;
    uint32_t     *leaf_id;
    float         lr;
    int           objective;
    float const  *labels;
    float2       *gh;
    uint32_t     *absmax;
    float const  *weights;
    TreeCommit    commit; // the finished tree's slot, or none
};

// The walk steps through the tree's decision heap (filled by the plan
// kernels): slot h's children are 2h + 1 and 2h + 2, so a step reads one
// 8-byte entry and no child ids. A leaf above the last level repeats down
// its left spine, and the slot a row ends in after `depth` steps names its
// leaf through leafmap.

__device__ __forceinline__ uint32_t heap_step(uint2 const e, uint32_t code, uint32_t h)
{
    bool const left = code <= (e.y & 0xFFFFu) || code == (e.y >> 16);
    return (2 * h) + (left ? 1u : 2u);
}

// A staged entry's x: the code's byte offset in the walking lane's column of the
// staged tile words (below 1,024), and the tile above it.
constexpr uint32_t k_no_staged_tile = k_no_tile & 0x3FFFFFu;

// The heap's entries and leaf map, staged in shared memory by the block.
template <bool U8>
__device__ __forceinline__ void load_heap(uint2 *heap_s, uint16_t *leaf_s, uint2 const *heap,
                                          uint16_t const *leafmap, uint32_t depth)
{
    uint32_t const n_int = (1u << depth) - 1;
    for (uint32_t i = threadIdx.x; i < n_int; i += blockDim.x)
    {
        uint2 const    e   = heap[i];
        uint32_t const pos = e.x & 0xFFu;
        uint32_t const off = U8 ? ((pos >> 2) * 128) + (pos & 3u)
                                : ((pos >> 1) * 128) + ((pos & 1u) * 2);
        heap_s[i]          = make_uint2(((e.x >> 8) << 10) | off, e.y);
    }
    for (uint32_t i = threadIdx.x; i <= n_int; i += blockDim.x)
    {
        leaf_s[i] = leafmap[i];
    }
    __syncthreads();
}

// Two rows' tiles in shared memory, word j of lane l's row at word 32 j + l of
// its warp's part, so a lane finds any code in its own bank.
__device__ __forceinline__ void stage_tile(uint32_t *col, uint4 const &a, uint4 const &b)
{
    uint32_t const w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
    for (uint32_t j = 0; j < 8; ++j)
    {
        col[32 * j] = w[j];
    }
}

// The last-level slots (leaf_s names their leaves) of a thread's two rows, step
// by step together: their tiles of the root's feature are staged; with MULTI
// the walk stages another tile when a slot's feature lives there. (Picked out
// of registers a code took a tree of selects, 30 instructions a step: pass A
// over 10,000,000 rows 135 us before, 113 now.)
template <bool U8, bool MULTI>
__device__ __forceinline__ void walk_heap(uint2 const *heap_s, uint32_t *col,
                                          uint4 const *__restrict__ mirror, uint64_t n_rows,
                                          uint64_t const (&r)[2], uint32_t depth, uint32_t held,
                                          uint32_t (&slot)[2])
{
    uint32_t const of[2]   = {0, 256};
    uint32_t       h[2]    = {0, 0};
    uint32_t       tile[2] = {held, held};
#pragma unroll
    for (uint32_t d = 0; d < 8; ++d)
    {
        if (d < depth)
        {
            uint2 e[2];
#pragma unroll
            for (uint32_t k = 0; k < 2; ++k)
            {
                e[k] = heap_s[h[k]];
                if constexpr (MULTI)
                {
                    uint32_t const t = e[k].x >> 10;
                    if (t != tile[k] && t != k_no_staged_tile)
                    {
                        uint4 const *src =
                            mirror + (((static_cast<uint64_t>(t) * n_rows) + r[k]) * 2);
                        stage_tile(col + of[k], src[0], src[1]);
                        tile[k] = t;
                    }
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < 2; ++k)
            {
                auto const *at = reinterpret_cast<unsigned char const *>(col + of[k]) +
                                 (e[k].x & 1023u);
                uint32_t const code = U8 ? *at : *reinterpret_cast<uint16_t const *>(at);
                h[k]                = heap_step(e[k], code, h[k]);
            }
        }
    }
    slot[0] = h[0] - ((1u << depth) - 1);
    slot[1] = h[1] - ((1u << depth) - 1);
}

// The tile that holds the root's feature (0 when the root is a leaf).
__device__ __forceinline__ uint32_t heap_root_tile(uint2 const *heap_s, uint32_t depth)
{
    uint32_t const t = depth > 0 ? heap_s[0].x >> 10 : k_no_staged_tile;
    return t == k_no_staged_tile ? 0u : t;
}

// Block maxima of |g| and h into the quantiser's two words.
__device__ __forceinline__ void block_absmax(float mg, float mh, uint32_t *absmax)
{
    __shared__ float mg_s[k_threads / 32];
    __shared__ float mh_s[k_threads / 32];
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        mg = fmaxf(mg, __shfl_xor_sync(0xFFFFFFFFu, mg, o));
        mh = fmaxf(mh, __shfl_xor_sync(0xFFFFFFFFu, mh, o));
    }
    if ((threadIdx.x & 31) == 0)
    {
        mg_s[threadIdx.x >> 5] = mg;
        mh_s[threadIdx.x >> 5] = mh;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (uint32_t w = 1; w < k_threads / 32; ++w)
        {
            mg = fmaxf(mg, mg_s[w]);
            mh = fmaxf(mh, mh_s[w]);
        }
        atomicMax(&absmax[0], __float_as_uint(mg));
        atomicMax(&absmax[1], __float_as_uint(mh));
    }
}

// A row's score update and, for a resident booster, its next gradient pair.
__device__ __forceinline__ void apply_leaf(WalkArgs const &a, uint64_t r, uint32_t leaf,
                                           float s_old, float y, float v, float &mg, float &mh)
{
    if (a.leaf_id != nullptr)
    {
        a.leaf_id[r] = leaf;
    }
    if (a.scores == nullptr)
    {
        return;
    }
    float const s = s_old + (a.lr * v);
    a.scores[r]   = s;
    if (a.gh != nullptr)
    {
        float2 const g = weighted(objective_gradient(a.objective, s, y), a.weights, r);
        a.gh[r]        = g;
        mg             = fmaxf(mg, fabsf(g.x));
        mh             = fmaxf(mh, fmaxf(g.y, 0.0F));
    }
}

// One pass: walk and apply (exact form), two rows per thread so their
// chains interleave.
template <bool U8, bool MULTI>
__global__ void __launch_bounds__(k_threads)
    walk_kernel(Ctl const *ctl, TreeOut t, uint4 const *__restrict__ mirror, uint64_t n_rows,
                uint2 const *heap, uint16_t const *leafmap, uint32_t depth, WalkArgs a)
{
    pdl_enter();
    __shared__ uint2    heap_s[k_heap_slots];
    __shared__ uint16_t leaf_s[k_heap_slots + 1];
    __shared__ float    val_s[k_walk_nodes];
    uint32_t const      n_nodes = min(ctl->n_nodes, k_walk_nodes);
    for (uint32_t i = threadIdx.x; i < n_nodes; i += k_threads)
    {
        val_s[i] = t.value[i];
    }
    __shared__ uint32_t codes_s[k_threads * 16];
    uint32_t *const     col = codes_s + ((threadIdx.x >> 5) * 512) + (threadIdx.x & 31);
    load_heap<U8>(heap_s, leaf_s, heap, leafmap, depth);
    uint32_t const root_tile = heap_root_tile(heap_s, depth);
    uint4 const   *mt        = mirror + (static_cast<uint64_t>(root_tile) * n_rows * 2);
    float          mg        = 0.0F;
    float          mh        = 0.0F;
    uint64_t const stride    = static_cast<uint64_t>(gridDim.x) * k_threads;
    uint64_t const pol       = l2_policy_first();
    for (uint64_t r0 = (static_cast<uint64_t>(blockIdx.x) * k_threads) + threadIdx.x;
         r0 < n_rows; r0 += 2 * stride)
    {
        uint64_t const r1  = r0 + stride;
        bool const     two = r1 < n_rows;
        uint64_t const rb  = two ? r1 : r0;
        uint4          a0, b0, a1, b1;
        ld_nc_row(mt + (r0 * 2), pol, a0, b0);
        ld_nc_row(mt + (rb * 2), pol, a1, b1);
        float const    s0  = a.scores != nullptr ? a.scores[r0] : 0.0F;
        float const    s1  = a.scores != nullptr ? a.scores[rb] : 0.0F;
        float const    y0  = a.gh != nullptr ? a.labels[r0] : 0.0F;
        float const    y1  = a.gh != nullptr ? a.labels[rb] : 0.0F;
        uint64_t const rr[2] = {r0, rb};
        uint32_t       o[2];
        stage_tile(col, a0, b0);
        stage_tile(col + 256, a1, b1);
        walk_heap<U8, MULTI>(heap_s, col, mirror, n_rows, rr, depth, root_tile, o);
        uint32_t const n0 = leaf_s[o[0]];
        uint32_t const n1 = leaf_s[o[1]];
        apply_leaf(a, r0, n0, s0, y0, val_s[n0], mg, mh);
        if (two)
        {
            apply_leaf(a, r1, n1, s1, y1, val_s[n1], mg, mh);
        }
    }
    if (a.absmax != nullptr)
    {
        block_absmax(mg, mh, a.absmax);
    }
    if (a.commit.round != nullptr && blockIdx.x == gridDim.x - 1)
    {
        commit_tree(t, a.commit);
    }
}

__device__ __forceinline__ bool in_sample(uint32_t const *bits, uint64_t r)
{
    return bits == nullptr || ((bits[r >> 5] >> (r & 31)) & 1u) != 0;
}

// Pass A of the quantised form: each row's leaf (as 16 bits) and every
// leaf's exact fixed-point (g, h) sums -- shared-memory 64-bit integer adds,
// then one global add per touched leaf and CTA. The shared sums are kept in
// k_wsum_copies lane-interleaved copies per last-level slot, laid out
// [slot][g, h][copy], so a warp's 64-bit adds -- copy = lane & 15 -- touch
// 16 distinct 8-byte words per half warp whatever slots its rows reach: two
// conflict-free wavefronts per add instead of one pass per row sharing a
// leaf. (Dynamic shared memory: 2^depth x 2 x 16 x 8 B.)
constexpr uint32_t k_wsum_thr    = 512;
constexpr uint32_t k_wsum_copies = 16;

// The quantised form's leaf values from pass A's sums: FP64 Newton values
// under each leaf's monotone bounds (one block). Run by pass A's last block,
// which then clears the gradients' maxima for the next round's where asked;
// a shard's sums are the fit's only after a reduction, so that it takes a
// launch of its own.
struct FixArgs
{
    Ctl const                *ctl;
    TreeOut                   t;
    unsigned long long const *acc;
    double2 const            *nbound;
    uint32_t const           *absmax;
    TreeParams                tp;
    double                    fix_unit;
    uint32_t                 *ticket; // null: not in pass A
    uint32_t                 *clear;  // the maxima to zero, or null
};

__device__ __forceinline__ void leaf_fix(FixArgs const &F)
{
    TreeOut const &t   = F.t;
    float const  mgx = __uint_as_float(F.absmax[0]);
    float const  mhx = __uint_as_float(F.absmax[1]);
    double const fg  = mgx > 0.0F ? F.fix_unit / static_cast<double>(mgx) : 1.0;
    double const fh  = mhx > 0.0F ? F.fix_unit / static_cast<double>(mhx) : 1.0;
    uint32_t const n_nodes = min(F.ctl->n_nodes, k_walk_nodes);
    for (uint32_t i = threadIdx.x; i < n_nodes; i += blockDim.x)
    {
        if (t.feature[i] != k_leaf_flag)
        {
            continue;
        }
        double const g = static_cast<double>(static_cast<int64_t>(F.acc[2 * i])) / fg;
        double const h = static_cast<double>(static_cast<int64_t>(F.acc[(2 * i) + 1])) / fh;
        double2 const b = F.nbound[i];
        t.value[i] = static_cast<float>(
            bounded_leaf_weight(g, h, F.tp.lambda_l1, F.tp.lambda_l2, b.x, b.y));
    }
}

template <bool U8, bool MULTI>
__global__ void __launch_bounds__(k_wsum_thr)
    walk_sum_kernel(Ctl const *ctl, uint4 const *__restrict__ mirror, uint64_t n_rows,
                    uint2 const *heap, uint16_t const *leafmap, uint32_t depth,
                    float2 const *__restrict__ gh, uint32_t const *absmax,
                    uint16_t *__restrict__ leaf16, unsigned long long *acc,
                    uint32_t const *__restrict__ bits, double fix_unit, FixArgs F)
{
    pdl_enter();
    extern __shared__ unsigned long long acc_s[];
    __shared__ uint2    heap_s[k_heap_slots];
    __shared__ uint16_t leaf_s[k_heap_slots + 1];
    uint32_t const      n_slot = 1u << depth;
    for (uint32_t i = threadIdx.x; i < n_slot * 2 * k_wsum_copies; i += k_wsum_thr)
    {
        acc_s[i] = 0ULL;
    }
    __shared__ uint32_t codes_s[k_wsum_thr * 16];
    uint32_t *const     col = codes_s + ((threadIdx.x >> 5) * 512) + (threadIdx.x & 31);
    load_heap<U8>(heap_s, leaf_s, heap, leafmap, depth);
    uint32_t const root_tile = heap_root_tile(heap_s, depth);
    uint4 const   *mt        = mirror + (static_cast<uint64_t>(root_tile) * n_rows * 2);
    float const    mgx       = __uint_as_float(absmax[0]);
    float const    mhx       = __uint_as_float(absmax[1]);
    double const   fg        = mgx > 0.0F ? fix_unit / static_cast<double>(mgx) : 1.0;
    double const   fh        = mhx > 0.0F ? fix_unit / static_cast<double>(mhx) : 1.0;
    uint64_t const stride    = static_cast<uint64_t>(gridDim.x) * k_wsum_thr;
    uint64_t const pol       = l2_policy_first();
    uint32_t const cp        = threadIdx.x & (k_wsum_copies - 1);
    auto           add       = [&](uint32_t o, float2 g)
    {
        uint32_t const x = (o * 2 * k_wsum_copies) + cp;
        atomicAdd(&acc_s[x],
                  static_cast<unsigned long long>(llrint(static_cast<double>(g.x) * fg)));
        atomicAdd(&acc_s[x + k_wsum_copies],
                  static_cast<unsigned long long>(
                      llrint(static_cast<double>(fmaxf(g.y, 0.0F)) * fh)));
    };
    for (uint64_t r0 = (static_cast<uint64_t>(blockIdx.x) * k_wsum_thr) + threadIdx.x;
         r0 < n_rows; r0 += 2 * stride)
    {
        uint64_t const r1  = r0 + stride;
        bool const     two = r1 < n_rows;
        uint64_t const rb  = two ? r1 : r0;
        uint4          a0, b0, a1, b1;
        ld_nc_row(mt + (r0 * 2), pol, a0, b0);
        ld_nc_row(mt + (rb * 2), pol, a1, b1);
        // a row outside this tree's sample takes its leaf but adds nothing
        float2 const   g0  = in_sample(bits, r0) ? gh[r0] : make_float2(0.0F, 0.0F);
        float2 const   g1  = in_sample(bits, rb) ? gh[rb] : make_float2(0.0F, 0.0F);
        uint64_t const rr[2] = {r0, rb};
        uint32_t       o[2];
        stage_tile(col, a0, b0);
        stage_tile(col + 256, a1, b1);
        walk_heap<U8, MULTI>(heap_s, col, mirror, n_rows, rr, depth, root_tile, o);
        uint32_t const o0 = o[0];
        uint32_t const o1 = o[1];
        leaf16[r0] = leaf_s[o0];
        add(o0, g0);
        if (two)
        {
            leaf16[r1] = leaf_s[o1];
            add(o1, g1);
        }
    }
    __syncthreads();
    // slot o's (g, h) over the copies, into its leaf's global sums (slots
    // that no row reaches hold zeros)
    for (uint32_t x = threadIdx.x; x < 2 * n_slot; x += k_wsum_thr)
    {
        unsigned long long v = 0ULL;
#pragma unroll
        for (uint32_t k = 0; k < k_wsum_copies; ++k)
        {
            v += acc_s[(x * k_wsum_copies) + k];
        }
        if (v != 0ULL)
        {
            atomicAdd(&acc[(2 * leaf_s[x >> 1]) + (x & 1)], v);
        }
    }
    if (F.ticket != nullptr && last_block(F.ticket, gridDim.x))
    {
        leaf_fix(F);
        __syncthreads();
        if (F.clear != nullptr && threadIdx.x < 2)
        {
            F.clear[threadIdx.x] = 0;
        }
    }
}

__global__ void __launch_bounds__(k_threads) leaf_fix_kernel(FixArgs F)
{
    pdl_enter();
    leaf_fix(F);
}

// Pass B of the quantised form: apply the renewed values by pass A's leaf ids.
__global__ void __launch_bounds__(k_threads)
    walk_apply_kernel(Ctl const *ctl, TreeOut t, uint64_t n_rows,
                      uint16_t const *__restrict__ leaf16, WalkArgs a)
{
    pdl_enter();
    __shared__ float val_s[k_walk_nodes];
    uint32_t const   n_nodes = min(ctl->n_nodes, k_walk_nodes);
    for (uint32_t i = threadIdx.x; i < n_nodes; i += k_threads)
    {
        val_s[i] = t.value[i];
    }
    __syncthreads();
    float          mg     = 0.0F;
    float          mh     = 0.0F;
    uint64_t const stride = static_cast<uint64_t>(gridDim.x) * k_threads;
    uint64_t const pol    = l2_policy_first(); // leaf ids, scores, labels: once a round
    for (uint64_t r = (static_cast<uint64_t>(blockIdx.x) * k_threads) + threadIdx.x; r < n_rows;
         r += stride)
    {
        uint32_t const n = ld_nc_u16(leaf16 + r, pol);
        float const    s = a.scores != nullptr ? __uint_as_float(ld_hint_b32(a.scores + r, pol))
                                               : 0.0F;
        float const    y = a.gh != nullptr ? __uint_as_float(ld_hint_b32(a.labels + r, pol))
                                           : 0.0F;
        apply_leaf(a, r, n, s, y, val_s[n], mg, mh);
    }
    if (a.absmax != nullptr)
    {
        block_absmax(mg, mh, a.absmax);
    }
    if (a.commit.round != nullptr && blockIdx.x == gridDim.x - 1)
    {
        commit_tree(t, a.commit);
    }
}

// Partition pass 2, the stable scatter: lefts keep their order at
// dst + left base, rights at dst + n_left + right base. Each warp takes the
// same run of rows as pass 1, its base from the bitmask's popcounts (one
// block barrier), its in-warp ranks from the bitmask words.
__global__ void __launch_bounds__(k_threads)
    pscatter_kernel(Ctl const *ctl, Chunk const *pchunks, Node const *nodes,
                    Best const *best, uint32_t const *pleft, uint32_t const *prbase,
                    uint32_t const *nleft, uint32_t const *dst,
                    uint32_t const *__restrict__ rows, uint32_t *__restrict__ rows_out,
                    uint32_t const *__restrict__ dirs, unsigned long long *zhist,
                    uint32_t const *build, uint32_t total_cells, uint32_t n_zcells)
{
    pdl_enter();
    __shared__ uint32_t wsum[k_threads / 32];
    uint32_t const      c = blockIdx.x;
    // the quantised build that follows adds into zeroed cells: every CTA
    // clears a share of the built slots' first n_zcells cells
    uint64_t const nz = static_cast<uint64_t>(ctl->n_build) * n_zcells;
    for (uint64_t x = (static_cast<uint64_t>(c) * k_threads) + threadIdx.x; x < nz;
         x += static_cast<uint64_t>(gridDim.x) * k_threads)
    {
        uint64_t const i = x / n_zcells;
        zhist[(static_cast<uint64_t>(build[i]) * total_cells) + (x - (i * n_zcells))] = 0ULL;
    }
    if (c >= ctl->n_pchunks)
    {
        return;
    }
    Chunk const ch = pchunks[c];
    Node const  nd = nodes[ch.node];
    if ((nd.flags & 1) == 0 || (nd.flags & 2) != 0)
    {
        return;
    }
    constexpr uint32_t steps = k_warp_rows / 32;
    uint32_t const     lane  = threadIdx.x & 31;
    uint32_t const     w     = threadIdx.x >> 5;
    uint32_t const     w0    = w * k_warp_rows;
    // the warp's direction words (lane i holds step i's) and row ids
    uint32_t const mword = lane < steps ? dirs[(static_cast<uint64_t>(c) * (k_part_rows / 32)) +
                                               (w * steps) + lane]
                                        : 0u;
    uint32_t r[steps];
#pragma unroll
    for (uint32_t i = 0; i < steps; ++i)
    {
        uint32_t const k = w0 + (32 * i) + lane;
        r[i]             = k < ch.count ? rows[ch.begin + k] : 0u;
    }
    // this warp's left count
    uint32_t mine = __popc(mword);
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        mine += __shfl_xor_sync(0xFFFFFFFFu, mine, o);
    }
    if (lane == 0)
    {
        wsum[w] = mine;
    }
    __syncthreads();
    uint32_t lb = 0;
    for (uint32_t x = 0; x < w; ++x)
    {
        lb += wsum[x];
    }
    uint32_t const d0  = dst[ch.node];
    uint32_t       lo  = d0 + pleft[c] + lb;                                   // next left
    uint32_t       ro  = d0 + nleft[ch.node] + prbase[c] + (min(w0, ch.count) - lb); // next right
    uint32_t const ltm = (1u << lane) - 1u;
#pragma unroll
    for (uint32_t i = 0; i < steps; ++i)
    {
        uint32_t const base = w0 + (32 * i);
        if (base >= ch.count)
        {
            break;
        }
        uint32_t const m      = __shfl_sync(0xFFFFFFFFu, mword, i);
        uint32_t const nvalid = min(32u, ch.count - base);
        uint32_t const vm     = nvalid == 32 ? 0xFFFFFFFFu : ((1u << nvalid) - 1u);
        uint32_t const lm     = m & vm;
        if (lane < nvalid)
        {
            if ((m >> lane) & 1u)
            {
                rows_out[lo + __popc(lm & ltm)] = r[i];
            }
            else
            {
                rows_out[ro + __popc(~lm & vm & ltm)] = r[i];
            }
        }
        lo += __popc(lm);
        ro += nvalid - __popc(lm);
    }
}

constexpr uint32_t k_psteps = k_warp_rows / 32; // 32-row steps of a partition warp

// One warp's 512 rows of a one-pass partition chunk: their ids (the level's
// list and the split column's codes are read once here, evict-first: the
// gradient codes and the next lists are what the level reads again) ...
template <bool FULL>
__device__ __forceinline__ void psplit_ids(Chunk const &ch, uint32_t const *__restrict__ rows,
                                           uint32_t w0, uint32_t lane, uint32_t (&r)[k_psteps])
{
    uint64_t const pol = l2_policy_first();
#pragma unroll
    for (uint32_t i = 0; i < k_psteps; ++i)
    {
        uint32_t const k = w0 + (32 * i) + lane;
        r[i]             = !FULL && k >= ch.count ? k_leaf_flag
                           : rows != nullptr      ? ld_hint_b32(rows + ch.begin + k, pol)
                                                  : ch.begin + k; // (the root's, every row)
    }
}

// ... their codes of the split feature, their directions (lane i keeps step
// i's bits).
template <bool FULL, typename BinT>
__device__ __forceinline__ void psplit_route(BinT const *col, uint4 const &route, uint32_t lane,
                                             uint32_t const (&r)[k_psteps], uint32_t &mword,
                                             uint32_t &n)
{
    uint64_t const pol = l2_policy_first();
    uint32_t       b[k_psteps];
#pragma unroll
    for (uint32_t i = 0; i < k_psteps; ++i)
    {
        b[i] = FULL || r[i] != k_leaf_flag ? ld_nc_code(col + r[i], pol) : 0u;
    }
#pragma unroll
    for (uint32_t i = 0; i < k_psteps; ++i)
    {
        bool const lf = (FULL || r[i] != k_leaf_flag) &&
                        routes_left(b[i], route.y, route.z, route.w != 0);
        uint32_t const m = __ballot_sync(0xFFFFFFFFu, lf);
        mword            = lane == i ? m : mword;
        n += __popc(m);
    }
}

// ... and their places: lefts from lo up, rights from top down (rank rk on).
template <bool FULL>
__device__ __forceinline__ void psplit_place(Chunk const &ch, uint32_t w0, uint32_t lane,
                                             uint32_t const (&r)[k_psteps], uint32_t mword,
                                             uint32_t lo, uint32_t rk, uint32_t top,
                                             uint32_t *__restrict__ rows_out)
{
    uint32_t const ltm = (1u << lane) - 1u;
#pragma unroll
    for (uint32_t i = 0; i < k_psteps; ++i)
    {
        uint32_t const base = w0 + (32 * i);
        if (!FULL && base >= ch.count)
        {
            break;
        }
        uint32_t const m      = __shfl_sync(0xFFFFFFFFu, mword, i);
        uint32_t const nvalid = FULL ? 32u : min(32u, ch.count - base);
        uint32_t const vm     = FULL || nvalid == 32 ? 0xFFFFFFFFu : ((1u << nvalid) - 1u);
        uint32_t const lm     = m & vm;
        if (FULL || lane < nvalid)
        {
            if ((m >> lane) & 1u)
            {
                rows_out[lo + __popc(lm & ltm)] = r[i];
            }
            else
            {
                rows_out[top - (rk + __popc(~lm & vm & ltm))] = r[i];
            }
        }
        lo += __popc(lm);
        rk += __popc(~lm & vm);
    }
}

// The partition in one pass, for trees the final walk stamps in the
// quantised form, whose every consumer of the row lists is order-free (the
// histogram build adds exact integers; the next partition routes row by
// row). Each chunk routes its rows as pcount_kernel does, then reserves its
// lefts' and rights' places in the node's own segment with one atomic add per
// side on per-node counters (zeroed by plan_kernel): lefts fill the segment
// from its start, rights from its end backwards, so pass 2, its re-read of the
// row ids and the chunk prefix sums in plan2_kernel fall away. Which chunk's
// rows come first inside a child depends on the order chunks finish; the
// histograms, splits and leaves do not. With SCATTER false (the last level,
// whose rows are never listed) only the left counts are taken. Also zeroes
// the next level's histogram slots [0, 2 x splits) for the build's adds.
template <typename BinT, bool SCATTER>
__global__ void __launch_bounds__(k_threads)
    psplit_kernel(Ctl const *ctl, Chunk const *pchunks, Node const *nodes, uint4 const *routes,
                  uint32_t const *__restrict__ rows, uint32_t *__restrict__ rows_out,
                  void const *__restrict__ bins, uint64_t n_pad, uint32_t *nleft, uint32_t *nright,
                  unsigned long long *zhist, uint32_t total_cells, uint32_t n_zcells)
{
    pdl_enter();
    __shared__ uint32_t wsum[k_threads / 32];
    __shared__ uint32_t base_s[2];
    uint32_t const      c    = blockIdx.x;
    Chunk const         ch   = pchunks[c]; // (a slot of the table, used or not)
    uint32_t const      n_ch = ctl->n_pchunks;
    uint32_t const      n_z  = ctl->n_psplit;
    uint32_t const      lane = threadIdx.x & 31;
    uint32_t const      w    = threadIdx.x >> 5;
    uint32_t const      w0   = w * k_warp_rows;
    // a warp whose 512 rows all lie in the chunk (the common case) skips the
    // per-row range checks
    bool const full = w0 + k_warp_rows <= ch.count;
    uint32_t   r[k_psteps];
    uint4      route{};
    uint32_t   start = 0;
    uint32_t   count = 0;
    bool       split = false;
    if (c < n_ch)
    {
        // the row ids, the node and its split all at once; a leaf's are unused
        full ? psplit_ids<true>(ch, rows, w0, lane, r) : psplit_ids<false>(ch, rows, w0, lane, r);
        route = routes[ch.node];
        start = nodes[ch.node].start;
        count = nodes[ch.node].count;
        split = (nodes[ch.node].flags & 1) != 0;
    }
    if constexpr (SCATTER)
    {
        uint64_t const nz = 2ULL * n_z * n_zcells;
        for (uint64_t x = (static_cast<uint64_t>(c) * k_threads) + threadIdx.x; x < nz;
             x += static_cast<uint64_t>(gridDim.x) * k_threads)
        {
            uint64_t const i = x / n_zcells;
            zhist[(i * total_cells) + (x - (i * n_zcells))] = 0ULL;
        }
    }
    if (!split)
    {
        return; // past the last chunk, or a leaf's, which routes nothing
    }
    BinT const *col   = static_cast<BinT const *>(bins) + (static_cast<uint64_t>(route.x) * n_pad);
    uint32_t    mword = 0; // lane i: step i's direction bits
    uint32_t    n     = 0;
    full ? psplit_route<true>(col, route, lane, r, mword, n)
         : psplit_route<false>(col, route, lane, r, mword, n);
    if (lane == 0)
    {
        wsum[w] = n;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        uint32_t lc = 0;
        for (uint32_t x = 0; x < k_threads / 32; ++x)
        {
            lc += wsum[x];
        }
        uint32_t const rc = ch.count - lc;
        base_s[0]         = lc != 0 ? atomicAdd(&nleft[ch.node], lc) : 0u;
        base_s[1]         = SCATTER && rc != 0 ? atomicAdd(&nright[ch.node], rc) : 0u;
    }
    if constexpr (!SCATTER)
    {
        return;
    }
    __syncthreads();
    uint32_t lb = 0;
    for (uint32_t x = 0; x < w; ++x)
    {
        lb += wsum[x];
    }
    uint32_t const lo  = start + base_s[0] + lb;                       // next left
    uint32_t const rk  = base_s[1] + (min(w0, ch.count) - lb);            // next right's rank
    uint32_t const top = start + count - 1;                          // rights count down
    if (full)
    {
        psplit_place<true>(ch, w0, lane, r, mword, lo, rk, top, rows_out);
    }
    else
    {
        psplit_place<false>(ch, w0, lane, r, mword, lo, rk, top, rows_out);
    }
}

constexpr uint32_t k_sub_cells = 1024; // cells per subtraction CTA

// Larger child = parent - smaller child, cell by cell in float
// (finish_split), 1,024 cells a block; both children's totals, summed from the
// same differences, and monotone bounds by each split's first block. (One block
// a split: 20.8 us a level of 28 features x 256 bins under ncu; now 9.0.)
__global__ void __launch_bounds__(k_threads)
    subtract_totals_kernel(Ctl *ctl, uint32_t const *bpair, float2 const *hist_cur,
                           float2 *hist_nxt, uint32_t total_cells, uint32_t n_cells,
                           Node const *cur, Node *next, Best const *best,
                           uint32_t const *sel, uint32_t const *sel_nb,
                           int8_t const *mono, uint32_t n_mono, TreeParams tp)
{
    pdl_enter();
    uint32_t const k = blockIdx.x;
    if (k == 0 && blockIdx.y == 0 && threadIdx.x == 0)
    {
        ctl->n_cur = ctl->n_next; // the level's last kernel advances the frontier
    }
    if (k >= ctl->n_splits)
    {
        return;
    }
    uint32_t const p  = bpair[3 * k];
    uint32_t const s  = bpair[(3 * k) + 1];
    uint32_t const l  = bpair[(3 * k) + 2];
    float2 const  *hp = hist_cur + (static_cast<uint64_t>(p) * total_cells);
    float2 const  *hs = hist_nxt + (static_cast<uint64_t>(s) * total_cells);
    float2        *hl = hist_nxt + (static_cast<uint64_t>(l) * total_cells);
    uint32_t const x0 = blockIdx.y * k_sub_cells;
    uint32_t const x1 = min(n_cells, x0 + k_sub_cells);
#pragma unroll 4
    for (uint32_t x = x0 + threadIdx.x; x < x1; x += k_threads)
    {
        float2 const a = hp[x];
        float2 const b = hs[x];
        hl[x]          = make_float2(a.x - b.x, a.y - b.y);
    }
    if (blockIdx.y != 0)
    {
        return;
    }
    // the children's totals: warp c sums child c's first feature
    __shared__ float tot_s[4];
    uint32_t const   wc = threadIdx.x >> 5;
    if (wc < 2)
    {
        float g, h;
        if ((2 * k) + wc == s)
        {
            warp_totals([&](uint32_t b) { return hs[b]; }, sel_nb[0], g, h);
        }
        else
        {
            warp_totals(
                [&](uint32_t b)
                {
                    float2 const a = hp[b];
                    float2 const c = hs[b];
                    return make_float2(a.x - c.x, a.y - c.y);
                },
                sel_nb[0], g, h);
        }
        if ((threadIdx.x & 31) == 0)
        {
            tot_s[2 * wc]       = g;
            tot_s[(2 * wc) + 1] = h;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        Node L  = next[2 * k];
        Node R  = next[(2 * k) + 1];
        L.sum_g = tot_s[0];
        L.sum_h = tot_s[1];
        R.sum_g = tot_s[2];
        R.sum_h = tot_s[3];
        Node const     par = cur[p];
        uint32_t const f   = sel[best[p].feature];
        int const      mc  = (mono != nullptr && f < n_mono) ? mono[f] : 0;
        if (mc != 0)
        {
            double const l1  = tp.lambda_l1;
            double const l2  = tp.lambda_l2;
            double const wl  = bounded_leaf_weight(L.sum_g, L.sum_h, l1, l2, par.lo, par.hi);
            double const wr  = bounded_leaf_weight(R.sum_g, R.sum_h, l1, l2, par.lo, par.hi);
            double const mid = 0.5 * (wl + wr);
            if (mc > 0)
            {
                L.hi = fmin(L.hi, mid);
                R.lo = fmax(R.lo, mid);
            }
            else
            {
                L.lo = fmax(L.lo, mid);
                R.hi = fmin(R.hi, mid);
            }
        }
        next[2 * k]       = L;
        next[(2 * k) + 1] = R;
    }
}

// The surviving frontier after the last level: leaves (end_tree). Marks
// every node a leaf and lays out its partition-chunk table, so the stamp
// (and, quantised, the leaf renewal) run chunk by chunk as on any level.
__global__ void __launch_bounds__(k_plan_thr)
    final_kernel(Ctl *ctl, Node *nodes, TreeParams tp, TreeOut t, Chunk *pchunks,
                 uint32_t *pcr, double2 *nbound, HeapOut ho, uint32_t *tree_no,
                 uint32_t tree_step)
{
    pdl_enter();
    uint32_t const n    = ctl->n_cur;
    uint32_t const i    = threadIdx.x;
    bool const     live = i < n;
    Node           nd   = live ? nodes[i] : Node{};
    if (live)
    {
        nbound[nd.id] = make_double2(nd.lo, nd.hi);
        write_leaf_node(t, nd.id, leaf_value(nd, tp));
        nd.flags = 0;
        nodes[i] = nd;
        heap_leaf(ho, nd.heap, nd.id);
    }
    uint32_t const nch   = live ? (nd.count + k_part_rows - 1) / k_part_rows : 0;
    uint32_t       total = 0;
    uint32_t const c0    = block_excl_scan<k_plan_thr>(nch, &total);
    if (live)
    {
        pcr[i] = c0;
    }
    if (i == 0)
    {
        pcr[n]          = total;
        ctl->n_pchunks  = total;
        ctl->n_leaves  += n;
        t.meta[0]       = ctl->n_nodes;
        t.meta[1]       = ctl->depth;
        t.meta[2]       = ctl->n_leaves;
        *tree_no       += tree_step; // (the tree's roundings are done)
    }
    __syncthreads();
    fill_chunk_table<k_plan_thr>(
        n, pcr, total, k_part_rows,
        [&](uint32_t x, uint32_t &st, uint32_t &cnt, uint32_t &aux)
        {
            Node const nx = nodes[x];
            st            = nx.start;
            cnt           = nx.count;
            aux           = 0;
        },
        pchunks);
}



// ------------------------------------------------------ quantised form ----
// Per tree: (g, h) scaled by FP64 scales max|g| / 127 and max h / 127 and
// stochastically rounded to int8 with a counter-based generator, so the
// histograms are exact integer sums (order-independent, deterministic). The
// split gain is evaluated in FP64 from the integer sums; leaf values are
// renewed in FP64 from the full-precision gradients of each leaf's rows
// (the scheme of Shi et al., "Quantized Training of Gradient Boosting
// Decision Trees", NeurIPS 2022).

// Philox4x32-10 (Salmon, Moraes, Dror and Shaw, "Parallel random numbers:
// as easy as 1, 2, 3", SC 2011): ten rounds of the Philox S-box with the
// published multipliers and Weyl key increments.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k)
{
    constexpr uint32_t m0 = 0xD2511F53u;
    constexpr uint32_t m1 = 0xCD9E8D57u;
    constexpr uint32_t w0 = 0x9E3779B9u;
    constexpr uint32_t w1 = 0xBB67AE85u;
#pragma unroll
    for (int r = 0; r < 10; ++r)
    {
        uint32_t const hi0 = __umulhi(m0, c.x);
        uint32_t const lo0 = m0 * c.x;
        uint32_t const hi1 = __umulhi(m1, c.z);
        uint32_t const lo1 = m1 * c.z;
        c                  = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
        k.x += w0;
        k.y += w1;
    }
    return c;
}

__global__ void __launch_bounds__(k_threads)
    absmax_kernel(float2 const *__restrict__ gh, uint32_t n, uint32_t *absmax)
{
    pdl_enter();
    __shared__ float sg[k_threads / 32];
    __shared__ float sh[k_threads / 32];
    float            mg = 0.0F;
    float            mh = 0.0F;
    for (uint32_t i = (blockIdx.x * k_threads) + threadIdx.x; i < n;
         i += gridDim.x * k_threads)
    {
        float2 const v = gh[i];
        mg             = fmaxf(mg, fabsf(v.x));
        mh             = fmaxf(mh, fmaxf(v.y, 0.0F));
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        mg = fmaxf(mg, __shfl_xor_sync(0xFFFFFFFFu, mg, o));
        mh = fmaxf(mh, __shfl_xor_sync(0xFFFFFFFFu, mh, o));
    }
    if ((threadIdx.x & 31) == 0)
    {
        sg[threadIdx.x >> 5] = mg;
        sh[threadIdx.x >> 5] = mh;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (uint32_t w = 1; w < k_threads / 32; ++w)
        {
            mg = fmaxf(mg, sg[w]);
            mh = fmaxf(mh, sh[w]);
        }
        // non-negative floats order as their bit patterns
        atomicMax(&absmax[0], __float_as_uint(mg));
        atomicMax(&absmax[1], __float_as_uint(mh));
    }
}

} // namespace

// What a tree starts with, done beside its quantisation (zero null: by
// launches of their own): the root's cells and the walk's sums zeroed, the root.
struct OpenArgs
{
    unsigned long long *zero;
    uint64_t            n_zero;
    unsigned long long *wacc;
    RootArgs            root;
};

namespace
{

// W16: int16 codes (scales max / 32767, g in the low half of a 32-bit word,
// h in the high half) instead of int8 (max / 127, a 16-bit word).
template <bool W16>
__global__ void __launch_bounds__(k_threads)
    quantise_kernel(float2 const *__restrict__ gh, uint32_t n,
                    uint32_t const *__restrict__ absmax, uint2 key,
                    uint32_t const *__restrict__ tree_no, void *__restrict__ qout,
                    double2 *__restrict__ scale, uint64_t row_off, OpenArgs O)
{
    pdl_enter();
    for (uint64_t x = (uint64_t{blockIdx.x} * k_threads) + threadIdx.x; x < O.n_zero;
         x += uint64_t{gridDim.x} * k_threads)
    {
        O.zero[x] = 0ULL;
    }
    if (O.zero != nullptr && blockIdx.x == gridDim.x - 1)
    {
        for (uint32_t x = threadIdx.x; x < 2 * k_walk_nodes; x += k_threads)
        {
            O.wacc[x] = 0ULL;
        }
        root_setup(O.root);
    }
    constexpr double qmax = W16 ? 32767.0 : 127.0;
    constexpr int    imax = W16 ? 32767 : 127;
    double const mg = __uint_as_float(absmax[0]);
    double const mh = __uint_as_float(absmax[1]);
    double const sg = mg > 0.0 ? mg / qmax : 1.0;
    double const sh = mh > 0.0 ? mh / qmax : 1.0;
    double const ig = 1.0 / sg; // one division per thread, a multiply per row
    double const ih = 1.0 / sh;
    uint32_t const t = *tree_no;
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        *scale = make_double2(sg, sh);
    }
    for (uint32_t i = (blockIdx.x * k_threads) + threadIdx.x; i < n;
         i += gridDim.x * k_threads)
    {
        float2 const v  = gh[i];
        // counter: the row's index in the whole fit, so shards round alike
        uint64_t const gi = row_off + i;
        uint4 const  r  = philox4x32_10(make_uint4(static_cast<uint32_t>(gi), t, 0x5157u,
                                                   static_cast<uint32_t>(gi >> 32)),
                                        key);
        double const ug = static_cast<double>(r.x >> 8) * (1.0 / 16777216.0);
        double const uh = static_cast<double>(r.y >> 8) * (1.0 / 16777216.0);
        double const xg = static_cast<double>(v.x) * ig;
        double const xh = static_cast<double>(fmaxf(v.y, 0.0F)) * ih;
        int          qg = isnan(xg) ? 0 : static_cast<int>(floor(xg + ug));
        int          qh = isnan(xh) ? 0 : static_cast<int>(floor(xh + uh));
        qg              = max(-imax, min(imax, qg));
        qh              = max(0, min(imax, qh));
        if constexpr (W16)
        {
            static_cast<uint32_t *>(qout)[i] =
                static_cast<uint32_t>(static_cast<uint16_t>(static_cast<int16_t>(qg))) |
                (static_cast<uint32_t>(qh) << 16);
        }
        else
        {
            static_cast<uint16_t *>(qout)[i] = static_cast<uint16_t>(
                static_cast<uint8_t>(static_cast<int8_t>(qg)) | (static_cast<uint32_t>(qh) << 8));
        }
    }
}

// Zeroes the cells of the nodes about to be built.
__global__ void __launch_bounds__(k_threads)
    zero_build_kernel(Ctl const *ctl, uint32_t const *build, unsigned long long *hist,
                      uint32_t total_cells, uint32_t n_cells)
{
    pdl_enter();
    uint32_t const i = blockIdx.x;
    if (i >= ctl->n_build)
    {
        return;
    }
    unsigned long long *h = hist + (static_cast<uint64_t>(build[i]) * total_cells);
    for (uint32_t x = threadIdx.x; x < n_cells; x += k_threads)
    {
        h[x] = 0ULL;
    }
}

// Exact integer histogram of a chunk of a built node's rows over one mirror
// tile: one gathered 32-byte sector per row, two native 32-bit
// shared-memory adds per (row, feature) -- the gradient word signed, the
// hessian word unsigned; a chunk's sums stay below 2^31 since a chunk holds
// at most 32,768 rows of |q| <= 127 -- then one packed 64-bit global add per
// touched cell (gradient in the high word, two's complement; hessian in the
// low word). grid (chunks, tiles), 256 threads.
// W16: int16 codes (a 32-bit word per row) into two-word cells (int64
// gradient, uint64 hessian sums); a 2,048-row chunk's sums of |q| <= 32767
// still fit the 32-bit shared words.
template <typename BinT, bool W16 = false, bool CW2 = W16>
__global__ void __launch_bounds__(k_qthreads, 3)
    qhist_kernel(Ctl const *ctl, Chunk const *bchunks, uint32_t const *build,
                 uint32_t const *rows, uint4 const *__restrict__ mirror, uint64_t n_rows,
                 void const *__restrict__ qgh, uint32_t const *tile_ids,
                 int32_t const *tile_j, uint32_t const *sel_nb, uint32_t const *cell_off,
                 uint32_t max_nb, unsigned long long *hist, uint32_t total_cells)
{
    pdl_enter();
    constexpr uint32_t per = k_mirror_bytes / sizeof(BinT);
    constexpr uint32_t U   = 2; // rows in flight per thread
    extern __shared__ int32_t hq_s[]; // [per][max_nb] gradient words, then hessian words
    __shared__ int32_t        j_s[per];
    uint32_t const            c = blockIdx.x;
    if (c >= ctl->n_bchunks)
    {
        return;
    }
    uint32_t const tile  = tile_ids[blockIdx.y];
    if (tile == k_no_sel_tile)
    {
        return; // a tile slot this selection leaves unused
    }
    uint32_t const cells = per * max_nb;
    int32_t       *hg_s  = hq_s;
    uint32_t      *hh_s  = reinterpret_cast<uint32_t *>(hq_s + cells);
    if (threadIdx.x < per)
    {
        j_s[threadIdx.x] = tile_j[(blockIdx.y * per) + threadIdx.x];
    }
    for (uint32_t x = threadIdx.x; x < 2 * cells; x += k_qthreads)
    {
        hq_s[x] = 0;
    }
    __syncthreads();
    Chunk const  ch = bchunks[c];
    uint4 const *mt = mirror + (static_cast<uint64_t>(tile) * n_rows * 2);
    for (uint32_t k0 = threadIdx.x; k0 < ch.count; k0 += k_qthreads * U)
    {
        uint32_t r[U];
        bool     ok[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u)
        {
            uint32_t const k = k0 + (u * k_qthreads);
            ok[u]            = k < ch.count;
            r[u]             = ok[u] ? (rows != nullptr ? rows[ch.begin + k] : ch.begin + k) : 0;
        }
        uint4    va[U];
        uint4    vb[U];
        uint32_t q[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u)
        {
            if (ok[u])
            {
                q[u]  = W16 ? static_cast<uint32_t const *>(qgh)[r[u]]
                            : static_cast<uint32_t>(static_cast<uint16_t const *>(qgh)[r[u]]);
                va[u] = mt[static_cast<uint64_t>(r[u]) * 2];
                vb[u] = mt[(static_cast<uint64_t>(r[u]) * 2) + 1];
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < U; ++u)
        {
            if (!ok[u])
            {
                continue;
            }
            int32_t const  qg   = W16 ? static_cast<int16_t>(q[u] & 0xFFFFu)
                                      : static_cast<int8_t>(q[u] & 0xFFu);
            uint32_t const qh   = W16 ? q[u] >> 16 : q[u] >> 8;
            uint32_t const w[8] = {va[u].x, va[u].y, va[u].z, va[u].w,
                                   vb[u].x, vb[u].y, vb[u].z, vb[u].w};
#pragma unroll
            for (uint32_t i = 0; i < per; ++i)
            {
                if (j_s[i] >= 0)
                {
                    uint32_t const bin =
                        sizeof(BinT) == 1 ? (w[i >> 2] >> ((i & 3) * 8)) & 0xFFu
                                          : (w[i >> 1] >> ((i & 1) * 16)) & 0xFFFFu;
                    uint32_t const x = (i * max_nb) + bin;
                    atomicAdd(&hg_s[x], qg);
                    atomicAdd(&hh_s[x], qh);
                }
            }
        }
    }
    __syncthreads();
    constexpr uint32_t  cw  = CW2 ? 2 : 1;
    unsigned long long *dst = hist + (static_cast<uint64_t>(build[ch.node]) * total_cells * cw);
    for (uint32_t x = threadIdx.x; x < cells; x += k_qthreads)
    {
        uint32_t const i  = x / max_nb;
        uint32_t const bb = x % max_nb;
        int32_t const  jj = j_s[i];
        if (jj >= 0 && bb < sel_nb[jj] && (hg_s[x] != 0 || hh_s[x] != 0))
        {
            uint64_t const cell = cell_off[jj] + bb;
            if constexpr (CW2)
            {
                atomicAdd(&dst[2 * cell],
                          static_cast<unsigned long long>(static_cast<int64_t>(hg_s[x])));
                atomicAdd(&dst[(2 * cell) + 1], static_cast<unsigned long long>(hh_s[x]));
            }
            else
            {
                atomicAdd(&dst[cell],
                          (static_cast<unsigned long long>(static_cast<uint32_t>(hg_s[x])) << 32) +
                              static_cast<unsigned long long>(hh_s[x]));
            }
        }
    }
}


// The u8 form of the quantised histogram, bank-conflict free without any
// staging: lane = row. At (unrolled) step i every lane handles feature
// i ^ lane of its row, so the 32 lanes touch 32 different features at every
// step. The shared table is [bin][g: 32 features][h: 32 features], 256 bytes
// per bin, so cell (b, f) sits in bank f whatever the bins, and its address
// is (b << 8) | (f << 2): one byte permute puts the row's code of feature
// i ^ lane at bits 8..15, one three-input logic op ORs in ((4 i) ^ (4 lane)),
// and two 32-bit shared reductions (gradient word signed, hessian word
// unsigned, at +0 and +128) complete the (row, feature). The 32-byte tile is
// brought into that order once per row by a word permutation (j -> j ^ lane/4,
// three select stages); the byte within a word is chosen by the permute's
// per-lane selector. Slots of unselected features accumulate into columns
// that are never flushed.
//
// Persistent: a grid of up to k_qctas CTAs per tile (one per SM; fewer for a
// small dataset, so several fits share the GPU), each walking a
// contiguous range of the level's chunks (node-ordered), so no wave tail.
// The loads are software-pipelined through registers: while a chunk's rows are
// added, the next chunk's codes and 32-byte tiles (one load a row), the row ids
// of the one after and the descriptor of the one after that are in flight, so
// that no load waits for the one that addresses it; the loop is unrolled by two
// so the prefetched registers are never moved (a move would wait for its
// load); with no shared staging the load/store path carries only the reductions
// (a reduction takes two cycles of it; the root's build is at 85% of that bound,
// the lower levels' wait for scattered DRAM sectors). 10,000,000 rows x 28, us:
// the root 132 before, 110 now, the next two levels 75 and 72, 60 and 70, the
// others as before; the round at 1,000,000 x depth 8 436 and 383. Shared memory
// beyond the table costs L1, which the loads in flight need (72 KB more: 96 to
// 108 us a level). The shared
// histogram flushes -- one packed 64-bit global add per touched cell,
// gradient in the high word (two's complement), hessian in the low word --
// only when the node changes. The 32-bit shared words cannot overflow in
// between: a CTA adds at most k_tshare_chunks chunks of 2,048 rows (the
// launch raises its CTA count to keep every share within that), so a word
// sums at most 16,908,288 codes of magnitude at most 127, below 2^31.
// Global cells are packed 64-bit words while 127 x the fit's rows stays
// below 2^31, and two words (int64 gradient, uint64 hessian sums, CW2)
// beyond that.
//
// The loads carry L2 eviction hints: the tiles are read once per build
// (evict-first), the 2-byte gradient codes by every build of the tree
// (evict-last), so below the root the codes are L2 hits instead of one
// random DRAM sector per built row.
constexpr uint32_t k_ttable_bytes = 256 * 256; // 256 bins x (32 g + 32 h) x 4 B
constexpr uint32_t k_tshare_chunks = 0x7FFFFFFFu / (127u * 2048u);


__device__ __forceinline__ void red_shared_u32(uint32_t addr, uint32_t v)
{
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

__device__ __forceinline__ void red_shared_u32_hi(uint32_t addr, uint32_t v)
{
    asm volatile("red.shared.add.u32 [%0+128], %1;" ::"r"(addr), "r"(v) : "memory");
}

// The table into the node's cells, and zeroed. Warp w takes bins [8w, 8w + 8):
// read lane = feature, turned in their own place so that eight lanes add one
// feature's eight consecutive cells (a lane per feature sent every add to a
// sector of its own: 8,192 a flush).
template <bool CW2>
__device__ __forceinline__ void qflush_t(uint32_t *tbl, uint32_t max_nb, uint32_t const *nb_s,
                                         uint32_t const *off_s, unsigned long long *dst)
{
    __syncthreads();
    uint32_t const lane = threadIdx.x & 31;
    uint32_t const b0   = (threadIdx.x >> 5) * 8;
    uint32_t      *mine = tbl + (b0 * 64);
    auto          *turn = reinterpret_cast<unsigned long long *>(mine);
    if (b0 < max_nb)
    {
        unsigned long long v[8];
#pragma unroll
        for (uint32_t b = 0; b < 8; ++b)
        {
            v[b] = (static_cast<unsigned long long>(mine[(b * 64) + lane]) << 32) |
                   mine[(b * 64) + 32 + lane];
        }
        __syncwarp();
#pragma unroll
        for (uint32_t b = 0; b < 8; ++b)
        {
            turn[(lane * 8) + (b ^ (lane & 7))] = v[b];
        }
        __syncwarp();
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q)
        {
            uint32_t const f = (q * 4) + (lane >> 3);
            v[q]             = turn[(f * 8) + ((lane ^ f) & 7)];
        }
        __syncwarp();
#pragma unroll
        for (uint32_t x = 0; x < 4; ++x)
        {
            reinterpret_cast<uint4 *>(mine)[(x * 32) + lane] = make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (uint32_t q = 0; q < 8; ++q)
        {
            uint32_t const f = (q * 4) + (lane >> 3);
            uint32_t const b = b0 + (lane & 7);
            if (v[q] != 0 && b < nb_s[f]) // (0 bins: not selected)
            {
                uint64_t const cell = off_s[f] + b;
                if constexpr (CW2)
                {
                    // two-word cells: the int64 gradient sum, the uint64 hessian sum
                    atomicAdd(&dst[2 * cell],
                              static_cast<unsigned long long>(static_cast<int64_t>(
                                  static_cast<int32_t>(static_cast<uint32_t>(v[q] >> 32)))));
                    atomicAdd(&dst[(2 * cell) + 1],
                              static_cast<unsigned long long>(static_cast<uint32_t>(v[q])));
                }
                else
                {
                    atomicAdd(&dst[cell], v[q]);
                }
            }
        }
    }
    __syncthreads();
}

// One row's 32 (feature, bin) cells: va, vb are the row's 32-byte tile.
__device__ __forceinline__ void qrow_t(uint32_t base, uint32_t lane4, uint32_t wsel,
                                       uint32_t const sel[4], uint4 va, uint4 vb, uint32_t q)
{
    uint32_t const qg = static_cast<uint32_t>(static_cast<int32_t>(static_cast<int8_t>(q & 0xFFu)));
    uint32_t const qh = q >> 8;
    uint32_t       w[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
#pragma unroll
    for (uint32_t st = 1; st < 8; st <<= 1)
    {
        bool const take = (wsel & st) != 0;
        uint32_t   t[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i)
        {
            t[i] = take ? w[i ^ st] : w[i];
        }
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i)
        {
            w[i] = t[i];
        }
    }
#pragma unroll
    for (uint32_t i = 0; i < 32; ++i)
    {
        uint32_t const off  = __byte_perm(w[i >> 2], 0u, sel[i & 3]) | ((4u * i) ^ lane4);
        uint32_t const addr = base + off;
        red_shared_u32(addr, qg);
        red_shared_u32_hi(addr, qh);
    }
}

constexpr uint32_t k_tper   = k_qbuild_rows / k_tthreads; // rows per thread per chunk
constexpr uint32_t k_tsmem  = k_ttable_bytes;               // the table
constexpr uint32_t k_no_row = 0xFFFFFFFFu;
static_assert(k_tper == 2, "the prefetch holds two rows per thread");

template <bool CW2>
__global__ void __launch_bounds__(k_tthreads, 1)
    qhist_t_kernel(Ctl const *ctl, Chunk const *bchunks, uint32_t const *build,
                   uint32_t const *__restrict__ rows, uint4 const *__restrict__ mirror,
                   uint64_t n_rows, uint16_t const *__restrict__ qgh, uint32_t const *tile_ids,
                   int32_t const *tile_j, uint32_t const *sel_nb, uint32_t const *cell_off,
                   uint32_t max_nb, unsigned long long *hist, uint32_t total_cells)
{
    pdl_enter();
    extern __shared__ uint4 t_smem[];
    __shared__ uint32_t     nb_s[32]; // per tile slot: its feature's bins (0: not selected)
    __shared__ uint32_t     off_s[32];
    uint32_t const          total = ctl->n_bchunks;
    uint32_t const          c_a   = static_cast<uint32_t>((static_cast<uint64_t>(blockIdx.x) * total) / gridDim.x);
    uint32_t const          c_b   = static_cast<uint32_t>((static_cast<uint64_t>(blockIdx.x + 1) * total) / gridDim.x);
    if (c_a >= c_b)
    {
        return;
    }
    uint32_t const tile = tile_ids[blockIdx.y];
    if (tile == k_no_sel_tile)
    {
        return; // a tile slot this selection leaves unused
    }
    uint32_t const tid  = threadIdx.x;
    uint32_t const lane = tid & 31;
    auto          *tbl  = reinterpret_cast<uint32_t *>(t_smem);
    uint32_t const base = static_cast<uint32_t>(__cvta_generic_to_shared(tbl));
    uint4 const   *mt    = mirror + (static_cast<uint64_t>(tile) * n_rows * 2);
    uint64_t const pol_t = l2_policy_first();
    uint64_t const pol_q = l2_policy_last();
    // a chunk's share of this thread: two rows, their codes and tiles
    struct Stage
    {
        uint32_t q[k_tper]; // k_no_row: no row
        uint4    a[k_tper];
        uint4    b[k_tper];
    };
    // a chunk, its row ids and its rows are each loaded an iteration apart, so
    // that none waits for the one it is addressed by
    auto const chunk = [&](uint32_t c) { return c < c_b ? bchunks[c] : Chunk{0, 0, 0, 0}; };
    auto const ids   = [&](Chunk const &ch, uint32_t id[k_tper])
    {
#pragma unroll
        for (uint32_t m = 0; m < k_tper; ++m)
        {
            uint32_t const k = (m * k_tthreads) + tid;
            id[m] = k < ch.count ? (rows != nullptr ? rows[ch.begin + k] : ch.begin + k)
                                 : k_no_row;
        }
    };
    auto const gather = [&](uint32_t const id[k_tper], Stage &S)
    {
#pragma unroll
        for (uint32_t m = 0; m < k_tper; ++m)
        {
            S.q[m] = k_no_row;
            if (id[m] != k_no_row)
            {
                uint4 const *src = mt + (static_cast<uint64_t>(id[m]) * 2);
                S.q[m]           = ld_nc_u16(qgh + id[m], pol_q);
                ld_nc_row(src, pol_t, S.a[m], S.b[m]);
            }
        }
    };
    Chunk    ch0 = chunk(c_a);     // of stage s0, then of the rows after s1's
    Chunk    ch1 = chunk(c_a + 1);
    uint32_t node  = ch0.node;
    uint32_t node0 = node;         // of s0's rows, of s1's
    uint32_t node1 = ch1.node;
    uint32_t id[k_tper];
    Stage    s0;
    Stage    s1;
    ids(ch0, id);
    gather(id, s0);
    ids(ch1, id);
    ch0 = chunk(c_a + 2);
    ch1 = chunk(c_a + 3);
    if (tid < 32)
    {
        int32_t const j = tile_j[(blockIdx.y * 32) + tid];
        nb_s[tid]       = j >= 0 ? sel_nb[j] : 0;
        off_s[tid]      = j >= 0 ? cell_off[j] : 0;
    }
    for (uint32_t x = tid; x < k_ttable_bytes / 16; x += k_tthreads)
    {
        t_smem[x] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    uint32_t sel[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
    {
        sel[k] = 0x4404u | (((k ^ lane) & 3u) << 4);
    }
    uint32_t const lane4 = lane * 4;
    uint32_t const wsel  = lane >> 2;
    auto           flush = [&]()
    {
        qflush_t<CW2>(tbl, max_nb, nb_s, off_s,
                      hist + (static_cast<uint64_t>(build[node]) * total_cells * (CW2 ? 2 : 1)));
    };
    auto run = [&](Stage const &S, uint32_t of)
    {
        if (of != node)
        {
            flush();
            node = of;
        }
#pragma unroll
        for (uint32_t m = 0; m < k_tper; ++m)
        {
            if (S.q[m] != k_no_row)
            {
                qrow_t(base, lane4, wsel, sel, S.a[m], S.b[m], S.q[m]);
            }
        }
    };
    for (uint32_t c = c_a; c < c_b; c += 2)
    {
        gather(id, s1); // chunk c + 1
        ids(ch0, id);   // c + 2
        uint32_t const n0 = ch0.node;
        ch0               = chunk(c + 4);
        run(s0, node0);
        if (c + 1 >= c_b)
        {
            break;
        }
        node0 = n0;
        gather(id, s0); // c + 2
        ids(ch1, id);   // c + 3
        uint32_t const n1 = ch1.node;
        ch1               = chunk(c + 5);
        run(s1, node1);
        node1 = n1;
    }
    flush();
}

__global__ void qroot_totals_kernel(Node *nodes, unsigned long long const *hist,
                                    uint32_t const *sel_nb, uint32_t cw)
{
    pdl_enter();
    int64_t g, h;
    warp_qtotals(hist, sel_nb[0], cw, g, h);
    if (threadIdx.x == 0)
    {
        nodes[0].qg = g;
        nodes[0].qh = h;
    }
}

// Larger child = parent - smaller child in exact integers (both packed
// words subtract without borrow: a child's hessian sum never exceeds its
// parent's); children's totals and monotone bounds from the integer sums.
__global__ void __launch_bounds__(k_threads)
    qsubtract_totals_kernel(Ctl *ctl, uint32_t const *bpair,
                            unsigned long long const *hist_cur, unsigned long long *hist_nxt,
                            uint32_t total_cells, uint32_t n_cells, Node const *cur,
                            Node *next, Best const *best, uint32_t const *sel,
                            uint32_t const *sel_nb, int8_t const *mono, uint32_t n_mono,
                            TreeParams tp, double2 const *qscale, int64_t const *btot,
                            uint32_t cw)
{
    pdl_enter();
    uint32_t const k = blockIdx.x;
    if (k == 0 && blockIdx.y == 0 && threadIdx.x == 0)
    {
        ctl->n_cur = ctl->n_next; // the level's last kernel advances the frontier
    }
    if (k >= ctl->n_splits)
    {
        return;
    }
    uint32_t const p  = bpair[3 * k];
    uint32_t const s  = bpair[(3 * k) + 1];
    uint32_t const l  = bpair[(3 * k) + 2];
    // words: cw per cell (two for int16 codes); the subtraction is word-wise
    auto const    *hp = hist_cur + (static_cast<uint64_t>(p) * total_cells * cw);
    auto const    *hs = hist_nxt + (static_cast<uint64_t>(s) * total_cells * cw);
    auto          *hl = hist_nxt + (static_cast<uint64_t>(l) * total_cells * cw);
    // blockIdx.y takes words [y * k_sub_cells, (y + 1) * k_sub_cells)
    uint32_t const x0 = blockIdx.y * k_sub_cells;
    uint32_t const x1 = min(n_cells * cw, x0 + k_sub_cells);
#pragma unroll 4
    for (uint32_t x = x0 + threadIdx.x; x < x1; x += k_threads)
    {
        hl[x] = hp[x] - hs[x];
    }
    if (blockIdx.y != 0 || threadIdx.x >= 32)
    {
        return;
    }
    // the smaller child's exact totals: its first feature's cells (every row
    // lands in one of them), or the per-build sums when no cells were built;
    // the larger child's are the parent's minus them
    int64_t sg = 0;
    int64_t sh = 0;
    if (btot != nullptr)
    {
        if (threadIdx.x == 0)
        {
            sg = btot[2 * k];
            sh = btot[(2 * k) + 1];
        }
    }
    else
    {
        for (uint32_t b = threadIdx.x; b < sel_nb[0]; b += 32)
        {
            int64_t cg, ch;
            qcell(hs, b, cw, cg, ch);
            sg += cg;
            sh += ch;
        }
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        sg += __shfl_xor_sync(0xFFFFFFFFu, sg, o);
        sh += __shfl_xor_sync(0xFFFFFFFFu, sh, o);
    }
    if (threadIdx.x == 0)
    {
        Node const par = cur[p];
        Node       S   = next[s];
        Node       G   = next[l];
        S.qg           = sg;
        S.qh           = sh;
        G.qg           = par.qg - sg;
        G.qh           = par.qh - sh;
        Node          &L  = s == 2 * k ? S : G;
        Node          &R  = s == 2 * k ? G : S;
        uint32_t const f  = sel[best[p].feature];
        int const      mc = (mono != nullptr && f < n_mono) ? mono[f] : 0;
        if (mc != 0)
        {
            split_bounds(L, R, par, mc, *qscale, tp);
        }
        next[2 * k]       = L;
        next[(2 * k) + 1] = R;
    }
}

// Exact integer totals of the smaller children when no histogram is built
// for them (the last level): per build chunk, the sums of its rows' codes,
// added into the chunk's build slot.
// The last level of a walked quantised tree: each built (smaller) child's
// exact integer totals straight from its parent's cells of the split
// feature -- the bins routes_left sends left (b <= split bin, and the missing
// bin when it defaults left), or the parent's totals minus them -- so the
// level needs neither the row scatter nor a gather of the children's codes.
// The parent's cells are the fit's (a sharded fit reduced them already).
// A warp per built child.
__global__ void qsplit_totals_kernel(Ctl const *ctl, uint32_t const *bpair, Node const *cur,
                                     Best const *best, unsigned long long const *hist_cur,
                                     uint32_t total_cells, uint32_t const *cell_off,
                                     uint32_t const *sel_nb, uint32_t cw, int64_t *btot)
{
    pdl_enter();
    uint32_t const k = (blockIdx.x * (blockDim.x / 32)) + (threadIdx.x >> 5);
    if (k >= ctl->n_splits)
    {
        return;
    }
    uint32_t const i       = bpair[3 * k];
    bool const     left_sm = (bpair[(3 * k) + 1] & 1u) == 0;
    Best const     b       = best[i];
    uint32_t const nb      = sel_nb[b.feature];
    uint32_t const last    = nb - 1;
    auto const    *cells   = hist_cur + (static_cast<uint64_t>(i) * total_cells * cw) +
                      (static_cast<uint64_t>(cell_off[b.feature]) * cw);
    int64_t lg = 0;
    int64_t lh = 0;
    for (uint32_t x = threadIdx.x & 31; x < nb; x += 32)
    {
        if (x == last ? b.dl != 0 : x <= b.bin)
        {
            int64_t cg, ch;
            qcell(cells, x, cw, cg, ch);
            lg += cg;
            lh += ch;
        }
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        lg += __shfl_xor_sync(0xFFFFFFFFu, lg, o);
        lh += __shfl_xor_sync(0xFFFFFFFFu, lh, o);
    }
    if ((threadIdx.x & 31) == 0)
    {
        Node const nd  = cur[i];
        btot[2 * k]     = left_sm ? lg : nd.qg - lg;
        btot[(2 * k) + 1] = left_sm ? lh : nd.qh - lh;
    }
}

__global__ void __launch_bounds__(k_threads)
    qbuilt_totals_kernel(Ctl const *ctl, Chunk const *bchunks, uint32_t const *rows,
                         uint16_t const *__restrict__ qgh, uint32_t const *__restrict__ qgh16,
                         int64_t *btot)
{
    pdl_enter();
    uint32_t const c = blockIdx.x;
    if (c >= ctl->n_bchunks)
    {
        return;
    }
    Chunk const ch = bchunks[c];
    int64_t     g  = 0;
    int64_t     h  = 0;
    for (uint32_t k = threadIdx.x; k < ch.count; k += k_threads)
    {
        uint32_t const r = rows[ch.begin + k];
        if (qgh16 != nullptr)
        {
            uint32_t const q = qgh16[r];
            g += static_cast<int16_t>(q & 0xFFFFu);
            h += q >> 16;
        }
        else
        {
            uint32_t const q = qgh[r];
            g += static_cast<int8_t>(q & 0xFFu);
            h += q >> 8;
        }
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        g += __shfl_xor_sync(0xFFFFFFFFu, g, o);
        h += __shfl_xor_sync(0xFFFFFFFFu, h, o);
    }
    if ((threadIdx.x & 31) == 0)
    {
        atomicAdd(reinterpret_cast<unsigned long long *>(&btot[2 * ch.node]),
                  static_cast<unsigned long long>(g));
        atomicAdd(reinterpret_cast<unsigned long long *>(&btot[(2 * ch.node) + 1]),
                  static_cast<unsigned long long>(h));
    }
}

// Leaf renewal: per partition chunk of a leaf node, the FP64 sums of the
// full-precision (g, h) of its rows in a fixed reduction order; the last CTA
// to finish (a ticket after a fence) then sums each leaf's chunks in chunk
// order and writes the FP64 Newton value under the node's bounds.
__global__ void __launch_bounds__(k_threads)
    leafsum_kernel(Ctl const *ctl, Chunk const *pchunks, Node const *nodes,
                   uint32_t const *__restrict__ rows, float2 const *__restrict__ gh,
                   double2 *partial, uint32_t const *pcr, TreeParams tp, TreeOut t,
                   uint32_t *done)
{
    pdl_enter();
    __shared__ double sg_s[k_threads / 32];
    __shared__ double sh_s[k_threads / 32];
    __shared__ bool   last_s;
    uint32_t const    c    = blockIdx.x;
    bool              work = c < ctl->n_pchunks;
    Chunk             ch{};
    if (work)
    {
        ch               = pchunks[c];
        Node const nd    = nodes[ch.node];
        work             = (nd.flags & 1) == 0 || (nd.flags & 2) != 0;
    }
    if (work)
    {
        double g = 0.0;
        double h = 0.0;
#pragma unroll 8
        for (uint32_t k = threadIdx.x; k < ch.count; k += k_threads)
        {
            float2 const v = gh[rows[ch.begin + k]];
            g += v.x;
            h += v.y;
        }
#pragma unroll
        for (uint32_t o = 16; o > 0; o >>= 1)
        {
            g += __shfl_xor_sync(0xFFFFFFFFu, g, o);
            h += __shfl_xor_sync(0xFFFFFFFFu, h, o);
        }
        if ((threadIdx.x & 31) == 0)
        {
            sg_s[threadIdx.x >> 5] = g;
            sh_s[threadIdx.x >> 5] = h;
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            double tg = 0.0;
            double th = 0.0;
            for (uint32_t w = 0; w < k_threads / 32; ++w)
            {
                tg += sg_s[w];
                th += sh_s[w];
            }
            partial[c] = make_double2(tg, th);
        }
    }
    if (threadIdx.x == 0)
    {
        __threadfence();
        last_s = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last_s)
    {
        return;
    }
    __threadfence();
    for (uint32_t i = threadIdx.x; i < ctl->n_cur; i += k_threads)
    {
        Node const nd = nodes[i];
        if ((nd.flags & 1) != 0 && (nd.flags & 2) == 0)
        {
            continue;
        }
        double g = 0.0;
        double h = 0.0;
        for (uint32_t x = pcr[i]; x < pcr[i + 1]; ++x)
        {
            double2 const v = __ldcg(&partial[x]);
            g += v.x;
            h += v.y;
        }
        t.value[nd.id] = static_cast<float>(
            bounded_leaf_weight(g, h, tp.lambda_l1, tp.lambda_l2, nd.lo, nd.hi));
    }
    if (threadIdx.x == 0)
    {
        *done = 0; // ready for the next launch
    }
}

// Larger child = parent - smaller, in place in the parent's slot (finish_split,
// float cells in float): the exact form's; the quantised form's pair kernel
// subtracts as it scans.
__global__ void leaf_sub_kernel(LeafOut const *out, uint32_t const *bpair, float2 *pool,
                                uint32_t total_cells, uint32_t n_cells)
{
    pdl_enter();
    if (out->split == 0)
    {
        return;
    }
    float2       *hp = pool + (static_cast<uint64_t>(bpair[0]) * total_cells);
    float2 const *hs = pool + (static_cast<uint64_t>(bpair[1]) * total_cells);
    for (uint32_t x = (blockIdx.x * blockDim.x) + threadIdx.x; x < n_cells;
         x += gridDim.x * blockDim.x)
    {
        float2 const a = hp[x];
        float2 const b = hs[x];
        hp[x]          = make_float2(a.x - b.x, a.y - b.y);
    }
}

// Both children's path state and monotone bounds (propagate_monotone_bounds,
// src/grower_impl.hpp:52-80) from their sums.
__device__ __forceinline__ void leaf_bounds(LeafPop const &p, uint32_t f, int mc,
                                            TreeParams const &tp, uint64_t const *fgroups,
                                            double gl, double hl, double gr, double hr, Node &L,
                                            Node &R)
{
    interaction_children(p.node, fgroups, f, L, R);
    if (mc != 0)
    {
        double const wl  = bounded_leaf_weight(gl, hl, tp.lambda_l1, tp.lambda_l2, p.node.lo,
                                               p.node.hi);
        double const wr  = bounded_leaf_weight(gr, hr, tp.lambda_l1, tp.lambda_l2, p.node.lo,
                                               p.node.hi);
        double const mid = 0.5 * (wl + wr);
        if (mc > 0)
        {
            L.hi = fmin(L.hi, mid);
            R.lo = fmax(R.lo, mid);
        }
        else
        {
            L.lo = fmax(L.lo, mid);
            R.hi = fmin(R.hi, mid);
        }
    }
}

// The children's totals from their cells (Histogram::totals), their path state
// and bounds: the exact form's.
__global__ void leaf_totals_kernel(Ctl *ctl, LeafOut const *out, Node *next,
                                   uint32_t const *slot_of, float2 const *pool,
                                   uint32_t total_cells, uint32_t const *sel,
                                   uint32_t const *sel_nb, int8_t const *mono, uint32_t n_mono,
                                   TreeParams tp, LeafPop const *pp, uint64_t const *fgroups)
{
    pdl_enter();
    __shared__ float tot_s[4];
    if (out->split == 0)
    {
        if (threadIdx.x == 0)
        {
            ctl->n_cur = 0;
        }
        return;
    }
    // warp c sums child c's first feature
    uint32_t const wc = threadIdx.x >> 5;
    if (wc < 2)
    {
        float g, h;
        float2 const *cells = pool + (static_cast<uint64_t>(slot_of[wc]) * total_cells);
        warp_totals([&](uint32_t b) { return cells[b]; }, sel_nb[0], g, h);
        if ((threadIdx.x & 31) == 0)
        {
            tot_s[2 * wc]       = g;
            tot_s[(2 * wc) + 1] = h;
        }
    }
    __syncthreads();
    if (threadIdx.x != 0)
    {
        return;
    }
    LeafPop const p = *pp;
    Node          L = next[0];
    Node          R = next[1];
    L.sum_g         = tot_s[0];
    L.sum_h         = tot_s[1];
    R.sum_g         = tot_s[2];
    R.sum_h         = tot_s[3];
    uint32_t const f = sel[p.best.feature];
    leaf_bounds(p, f, (mono != nullptr && f < n_mono) ? mono[f] : 0, tp, fgroups, L.sum_g, L.sum_h,
                R.sum_g, R.sum_h, L, R);
    next[0]    = L;
    next[1]    = R;
    ctl->n_cur = 2;
}

// Each node's best split over the features (the lowest feature wins a gain
// tie), no split past the depth cap: the root's, and the exact form's pairs'.
// grid 2 (a CTA per node) x k_best_thr: each thread scans a stride of the
// features, then (largest gain, lowest feature) over the block -- the serial
// scan's choice, whatever the order.
constexpr uint32_t k_best_thr = 256;

__global__ void __launch_bounds__(k_best_thr)
    leaf_best_kernel(Ctl const *ctl, Best const *cand, uint32_t n_sel, Node const *nodes,
                     LeafOut *out, uint32_t const *may_split_p)
{
    pdl_enter();
    uint32_t const      may_split = *may_split_p;
    __shared__ double   g_s[k_best_thr / 32];
    __shared__ uint32_t o_s[k_best_thr / 32];
    uint32_t const      w    = blockIdx.x;
    uint32_t const      lane = threadIdx.x & 31;
    bool const          live = w < ctl->n_cur;
    double              g    = 0.0;
    uint32_t            o    = 0xFFFFFFFFu;
    for (uint32_t j = threadIdx.x; live && may_split != 0 && j < n_sel; j += k_best_thr)
    {
        Best const c = cand[(w * n_sel) + j];
        if (c.valid != 0 && (c.gain > g || (c.gain == g && j < o)))
        {
            g = c.gain;
            o = j;
        }
    }
    warp_best(g, o);
    if (lane == 0)
    {
        g_s[threadIdx.x >> 5] = g;
        o_s[threadIdx.x >> 5] = o;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (uint32_t x = 1; x < k_best_thr / 32; ++x)
        {
            if (g_s[x] > g || (g_s[x] == g && o_s[x] < o))
            {
                g = g_s[x];
                o = o_s[x];
            }
        }
        out->best[w] = o == 0xFFFFFFFFu ? Best{0.0, 0, 0, 1, 0} : cand[(w * n_sel) + o];
        if (live)
        {
            out->child[w] = nodes[w];
        }
    }
}

// ---- the leafwise pop loop on the device -----------------------------------
// LeafwiseGrower::grow's heap loop (src/grower_impl.hpp:744-850): the gain
// max-heap (ties to the lower node id, so growth is deterministic), the
// histogram pool's free slots, the node table and the leaf list all live on
// the device, and one pop is a fixed sequence of launches that a CUDA graph's
// conditional WHILE node repeats until the heap is empty or the leaf budget
// is spent -- no host round trip per pop.

struct LeafCand
{
    Node     node;
    Best     best;
    uint32_t depth;
    uint32_t slot;
};

struct LeafLoop
{
    LeafPop  pop;        // the current pop
    uint32_t pop_depth;
    uint32_t may_split;  // the pop's children may split (depth cap)
    uint32_t root_may;   // the root may split
    uint32_t noop;       // nothing was popped
    uint32_t n_cand;
    uint32_t n_leaves;
    uint32_t n_nodes;
    uint32_t live;
    uint32_t depth;
    uint32_t n_free;
    uint32_t error;      // 1: the node table is full, 2: the histogram pool is
    uint32_t pops;       // pops taken this tree
};

// After the root's find: the root a candidate (or a leaf), the node table's
// first entry, every pool slot but the root's free.
__global__ void __launch_bounds__(k_plan_thr)
    leaf_loop_init_kernel(LeafLoop *st, LeafCand *cand, Node *leaves, uint32_t *free_slots,
                          LeafOut const *out, TreeOut const *tp_, uint32_t n_root,
                          uint32_t max_front, uint32_t max_depth)
{
    pdl_enter();
    for (uint32_t k = threadIdx.x; k + 1 < max_front; k += k_plan_thr)
    {
        free_slots[k] = max_front - 1 - k; // popped from the top: slot 1 first
    }
    if (threadIdx.x != 0)
    {
        return;
    }
    TreeOut const t   = *tp_;
    t.feature[0]      = k_leaf_flag;
    t.left[0]         = 0;
    t.right[0]        = 0;
    t.split_bin[0]    = 0;
    t.value[0]        = 0.0F;
    t.gain[0]         = 0.0F;
    t.cover[0]        = static_cast<float>(n_root);
    t.default_left[0] = 0;
    LeafCand const root{out->child[0], out->best[0], 0, 0};
    bool const     ok = root.best.valid != 0 && max_depth > 0;
    st->n_cand        = ok ? 1 : 0;
    if (ok)
    {
        cand[0] = root;
    }
    else
    {
        leaves[0] = root.node;
    }
    st->n_leaves = ok ? 0 : 1;
    st->n_nodes  = 1;
    st->live     = 1;
    st->depth    = 0;
    st->n_free   = max_front - 1;
    st->error    = 0;
    st->pops     = 0;
    st->noop     = 0;
}

// What the loop's turns work on.
struct LeafTurn
{
    LeafLoop       *st;
    LeafCand       *cand;
    Node           *leaves;
    uint32_t       *free_slots;
    LeafOut        *out;
    TreeOut const  *tree;
    float const    *cuts;
    uint32_t const *cut_off, *sel;
    uint32_t        max_leaves, max_nodes, max_depth, max_pops;
    Ctl            *ctl;
    Node           *nodes;
    Best           *best;
    Chunk          *pchunks;
    uint32_t       *pcr;
};

// One pop, by a CTA of k_pop_thr threads: the best candidate off the heap,
// commit_split_node (src/grower_impl.hpp:189-206) into the node table, a pool
// slot for the smaller child, and the popped node's partition chunks (the
// setup of one pop). With nothing to pop it sets the no-op flag and leaves no
// chunks and no split, so that an iteration after it does nothing (a tree that
// is its root alone still runs the loop's body once, and without chunks no
// CTA of it plans children). Returns whether it popped.
constexpr uint32_t k_pop_thr = 256;

__device__ __forceinline__ bool leaf_pop(LeafTurn const &T)
{
    __shared__ double   g_s[k_pop_thr / 32];
    __shared__ uint32_t id_s[k_pop_thr / 32];
    __shared__ uint32_t ix_s[k_pop_thr / 32];
    __shared__ uint32_t go_s;
    uint32_t const      n    = T.st->n_cand;
    uint32_t const      lane = threadIdx.x & 31;
    if (threadIdx.x == 0)
    {
        bool const go = T.st->error == 0 && n > 0 && (T.max_leaves == 0 || T.st->live < T.max_leaves);
        go_s          = go ? 1 : 0;
        T.st->noop      = go ? 0 : 1;
        if (!go)
        {
            T.ctl->n_cur     = 0;
            T.ctl->n_pchunks = 0;
            T.ctl->n_build   = 0;
            T.ctl->n_bchunks = 0;
            T.pcr[0]         = 0;
            T.pcr[1]         = 0;
            T.out->split     = 0;
            T.st->pop.node.count = 0;
        }
    }
    __syncthreads();
    if (go_s == 0)
    {
        return false;
    }
    // the heap's top: the largest gain, then the lowest node id
    double   g  = -1.0;
    uint32_t id = 0xFFFFFFFFu;
    uint32_t ix = 0;
    for (uint32_t i = threadIdx.x; i < n; i += k_pop_thr)
    {
        double const   cg  = T.cand[i].best.gain;
        uint32_t const cid = T.cand[i].node.id;
        if (cg > g || (cg == g && cid < id))
        {
            g  = cg;
            id = cid;
            ix = i;
        }
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        double const   og  = __shfl_xor_sync(0xFFFFFFFFu, g, o);
        uint32_t const oid = __shfl_xor_sync(0xFFFFFFFFu, id, o);
        uint32_t const oix = __shfl_xor_sync(0xFFFFFFFFu, ix, o);
        if (og > g || (og == g && oid < id))
        {
            g  = og;
            id = oid;
            ix = oix;
        }
    }
    if (lane == 0)
    {
        g_s[threadIdx.x >> 5]  = g;
        id_s[threadIdx.x >> 5] = id;
        ix_s[threadIdx.x >> 5] = ix;
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        for (uint32_t w = 1; w < k_pop_thr / 32; ++w)
        {
            if (g_s[w] > g || (g_s[w] == g && id_s[w] < id))
            {
                g  = g_s[w];
                id = id_s[w];
                ix = ix_s[w];
            }
        }
        LeafCand const c = T.cand[ix];
        T.cand[ix]         = T.cand[n - 1];
        T.st->n_cand       = n - 1;
        uint32_t const lid = T.st->n_nodes;
        uint32_t const rid = lid + 1;
        if (rid >= T.max_nodes || T.st->n_free == 0)
        {
            T.st->error          = rid >= T.max_nodes ? 1 : 2;
            T.st->noop           = 1;
            T.ctl->n_cur         = 0;
            T.ctl->n_pchunks     = 0;
            T.ctl->n_build       = 0;
            T.ctl->n_bchunks     = 0;
            T.pcr[0]             = 0;
            T.pcr[1]             = 0;
            T.out->split         = 0;
            T.st->pop.node.count = 0;
            go_s               = 0;
        }
        else
        {
            TreeOut const t = *T.tree;
            for (uint32_t k = lid; k <= rid; ++k)
            {
                t.feature[k]      = k_leaf_flag;
                t.left[k]         = 0;
                t.right[k]        = 0;
                t.split_bin[k]    = 0;
                t.value[k]        = 0.0F;
                t.gain[k]         = 0.0F;
                t.cover[k]        = 0.0F;
                t.default_left[k] = 0;
            }
            uint32_t const f     = T.sel[c.best.feature];
            uint32_t const nid   = c.node.id;
            t.feature[nid]       = f;
            t.value[nid]         = T.cuts[T.cut_off[f] + c.best.bin];
            t.left[nid]          = lid;
            t.right[nid]         = rid;
            t.default_left[nid]  = static_cast<uint8_t>(c.best.dl);
            t.gain[nid]          = static_cast<float>(c.best.gain);
            t.split_bin[nid]     = c.best.bin;
            T.st->n_nodes          = rid + 1;
            uint32_t const small = T.free_slots[--T.st->n_free];
            T.st->pop       = LeafPop{c.node, c.best, lid, rid, c.slot, small};
            T.st->pop_depth = c.depth;
            T.st->may_split = c.depth + 1 < T.max_depth ? 1 : 0;
            T.st->pops += 1;
            // the pop's setup: the node's partition chunks
            uint32_t const nch = (c.node.count + k_part_rows - 1) / k_part_rows;
            T.ctl->n_cur         = 1;
            T.ctl->n_pchunks     = nch;
            Node nd            = c.node;
            nd.flags           = 1;
            T.nodes[0]           = nd;
            T.best[0]            = c.best;
            T.pcr[0]             = 0;
            T.pcr[1]             = nch;
        }
    }
    __syncthreads();
    if (go_s == 0)
    {
        return false;
    }
    LeafPop const &p   = T.st->pop;
    uint32_t const cnt = p.node.count;
    uint32_t const nch = (cnt + k_part_rows - 1) / k_part_rows;
    for (uint32_t c = threadIdx.x; c < nch; c += k_pop_thr)
    {
        uint32_t const b = c * k_part_rows;
        T.pchunks[c]       = {0, p.node.start + b, min(k_part_rows, cnt - b), 0};
    }
    return true;
}

// The last pop's outcome into the loop's state, by one thread: commit_pop's
// demotion, or the two children queued (queue_children,
// src/grower_impl.hpp:405-425).
__device__ __forceinline__ void leaf_commit(LeafTurn const &T)
{
    LeafLoop      *st = T.st;
    LeafPop const &p  = st->pop;
    TreeOut const  t  = *T.tree;
    if (T.out->split == 0)
    {
        // the survivor holds the parent's rows and takes its id and bounds; the
        // two children stay placeholders
        t.gain[p.node.id]          = 0.0F;
        T.leaves[st->n_leaves++]   = p.node;
        T.free_slots[st->n_free++] = p.small_slot;
        T.free_slots[st->n_free++] = p.parent_slot;
    }
    else
    {
        Node const     L  = T.out->child[0];
        Node const     R  = T.out->child[1];
        bool const     sl = T.out->small_left != 0;
        uint32_t const d  = st->pop_depth + 1;
        t.cover[p.left_id]  = static_cast<float>(L.gcount);
        t.cover[p.right_id] = static_cast<float>(R.gcount);
        st->live += 1;
        st->depth = max(st->depth, d);
        LeafCand const kids[2] = {{L, T.out->best[0], d, sl ? p.small_slot : p.parent_slot},
                                  {R, T.out->best[1], d, sl ? p.parent_slot : p.small_slot}};
        for (LeafCand const &k : kids)
        {
            if (k.best.valid != 0)
            {
                T.cand[st->n_cand++] = k;
            }
            else
            {
                T.leaves[st->n_leaves++]   = k.node;
                T.free_slots[st->n_free++] = k.slot;
            }
        }
    }
    // every pop either adds a leaf or retires a candidate, so at most
    // 2 x max_leaves pops ever run; past max_pops the loop stops with an error
    // rather than spin
    if (st->pops >= T.max_pops)
    {
        st->error = 3;
    }
}

// A turn of the loop, by a CTA: the last pop's outcome, the next pop, and
// whether the loop goes on. One CTA does both, in a launch where each had its
// own.
__device__ __forceinline__ void leaf_turn(LeafTurn const &T, cudaGraphConditionalHandle handle)
{
    if (threadIdx.x == 0 && T.st->noop == 0)
    {
        leaf_commit(T);
    }
    __syncthreads();
    bool const more = leaf_pop(T);
    if (threadIdx.x == 0)
    {
        cudaGraphSetConditional(handle, more ? 1u : 0u);
    }
}

// The tree's first pop, before the loop.
__global__ void __launch_bounds__(k_pop_thr) leaf_first_pop_kernel(LeafTurn T)
{
    pdl_enter();
    leaf_pop(T);
}

// The exact form's turn, after its find.
__global__ void __launch_bounds__(k_pop_thr)
    leaf_turn_kernel(LeafTurn T, cudaGraphConditionalHandle handle)
{
    pdl_enter();
    leaf_turn(T, handle);
}

// A pop's second half in the quantised form, in one launch where five had
// their own: the larger child = parent - smaller, in place in the parent's
// slot (integer words subtract without borrow), both children's totals,
// bounds and best splits, and the turn of the loop. Two warps per feature,
// one per child; the larger child's cells come straight from the subtraction,
// and a node's totals are that feature's own sums (exact integers, the same
// for every feature). The warps' choices are reduced per CTA, and the last CTA
// reduces those and takes the turn. (Two CTAs an SM: held to 128 registers
// two-word cells spill one, and a round of 100,000 rows x 2,000 int16 takes
// 20.4 ms; with 152 and one CTA an SM 22.8.)
template <bool CW2>
__global__ void __launch_bounds__(k_pop_thr, 2)
    leaf_pair_kernel(LeafTurn T, LeafOut *out, Node const *next, unsigned long long *pool,
                     uint32_t total_cells, uint32_t const *cell_off, uint32_t const *sel_nb,
                     uint32_t n_sel, int8_t const *mono, uint32_t n_mono, TreeParams tp,
                     double2 const *qscale, uint64_t const *fgroups, Best *part,
                     uint32_t *ticket, cudaGraphConditionalHandle handle)
{
    pdl_enter();
    constexpr uint32_t warps = k_pop_thr / 32;
    constexpr uint32_t cw    = CW2 ? 2 : 1;
    __shared__ QHand<CW2> hand_s[warps];
    __shared__ double     g_s[warps];
    __shared__ uint32_t   o_s[warps];
    __shared__ uint32_t   j_s[warps];
    __shared__ bool       last_s;
    LeafLoop const       *st = T.st;
    uint32_t const      lane = threadIdx.x & 31;
    uint32_t const      w    = threadIdx.x >> 5;
    bool const          work = st->noop == 0 && out->split != 0;
    if (work)
    {
        LeafPop const &p     = st->pop;
        uint32_t const j     = (blockIdx.x * (warps / 2)) + (w >> 1);
        bool const     large = (w & 1) != 0;
        // this warp's child: 0 left, 1 right
        uint32_t const x     = (out->small_left != 0) != large ? 0 : 1;
        double         best  = 0.0;
        uint32_t       order = 0xFFFFFFFFu;
        if (j < n_sel)
        {
            uint32_t const nb = sel_nb[j];
            auto const    *hs = pool +
                             (((static_cast<uint64_t>(p.small_slot) * total_cells) + cell_off[j]) * cw);
            auto *hp = pool +
                       (((static_cast<uint64_t>(p.parent_slot) * total_cells) + cell_off[j]) * cw);
            bool const held = nb <= 32 * k_qfind_group; // every bin in registers at once
            QCell<CW2> v[k_qfind_group];
            QCell<CW2> carry, before, miss;
            carry.clear();
            auto load = [&](uint32_t c0)
            {
#pragma unroll
                for (uint32_t q = 0; q < k_qfind_group; ++q)
                {
                    uint32_t const b = c0 + (q * 32) + lane;
                    v[q].clear();
                    if (b < nb)
                    {
                        v[q].load(large ? hp : hs, b);
                    }
                }
                if (large)
                {
                    QCell<CW2> u[k_qfind_group];
#pragma unroll
                    for (uint32_t q = 0; q < k_qfind_group; ++q)
                    {
                        uint32_t const b = c0 + (q * 32) + lane;
                        u[q].clear();
                        if (b < nb)
                        {
                            u[q].load(hs, b);
                        }
                    }
#pragma unroll
                    for (uint32_t q = 0; q < k_qfind_group; ++q)
                    {
                        uint32_t const b = c0 + (q * 32) + lane;
                        v[q].sub(u[q]);
                        if (b < nb)
                        {
                            v[q].store(hp, b);
                        }
                    }
                }
            };
            // the child's totals and its missing bin
            int64_t qg = 0;
            int64_t qh = 0;
            miss.load(hs, nb - 1);
            if (large)
            {
                QCell<CW2> m;
                m.load(hp, nb - 1);
                m.sub(miss);
                miss = m;
            }
            if (held)
            {
                __syncwarp(); // (the missing bin is read before it is rewritten)
                load(0);
                qscan_group<CW2>(v, hand_s[w], carry, before);
                qg = carry.g();
                qh = carry.h();
            }
            else
            {
                warp_qtotals(hs, nb, cw, qg, qh);
                qg = large ? p.node.qg - qg : qg;
                qh = large ? p.node.qh - qh : qh;
                __syncwarp();
            }
            double2 const  sc   = *qscale;
            Node           nd   = next[x]; // this child, and what its bounds take of its sibling
            Node           sib  = next[x ^ 1];
            nd.qg               = qg;
            nd.qh               = qh;
            uint32_t const pf   = T.sel[p.best.feature];
            double const   g    = static_cast<double>(qg) * sc.x;
            double const   h    = static_cast<double>(qh) * sc.y;
            double const   sg   = static_cast<double>(p.node.qg - qg) * sc.x;
            double const   sh   = static_cast<double>(p.node.qh - qh) * sc.y;
            int const      pmc  = (mono != nullptr && pf < n_mono) ? mono[pf] : 0;
            if (x == 0)
            {
                leaf_bounds(p, pf, pmc, tp, fgroups, g, h, sg, sh, nd, sib);
            }
            else
            {
                leaf_bounds(p, pf, pmc, tp, fgroups, sg, sh, g, h, sib, nd);
            }
            if (j == 0 && lane == 0)
            {
                out->child[x] = nd;
                __threadfence();
            }
            uint32_t const f = T.sel[j];
            bool const may = st->may_split != 0 && nd.gcount >= 2 * tp.min_data_in_leaf && nb >= 2 &&
                             interaction_allows(nd, fgroups, f);
            QNode n;
            n.start(qg, qh, miss.g(), miss.h(), nd, (mono != nullptr && f < n_mono) ? mono[f] : 0,
                    sc, tp, CW2 ? 32767.0F : 127.0F);
            if (held)
            {
                if (may)
                {
                    qscore_group<CW2>(v, before, 0, nb - 2, n, sc, tp, best, order);
                }
            }
            else
            {
                for (uint32_t c0 = 0; c0 < nb; c0 += 32 * k_qfind_group)
                {
                    load(c0);
                    qscan_group<CW2>(v, hand_s[w], carry, before);
                    if (may)
                    {
                        qscore_group<CW2>(v, before, c0, nb - 2, n, sc, tp, best, order);
                    }
                }
            }
        }
        warp_best(best, order);
        if (lane == 0)
        {
            g_s[w] = best;
            o_s[w] = order;
            j_s[w] = j;
        }
        __syncthreads();
        if (threadIdx.x < 2)
        {
            // features in order: a later one has to gain more
            uint32_t const lg = threadIdx.x; // the smaller or the larger child
            Best           b  = {0.0, 0, 0, 1, 0};
            for (uint32_t u = lg; u < warps; u += 2)
            {
                if (o_s[u] != 0xFFFFFFFFu && (b.valid == 0 || g_s[u] > b.gain))
                {
                    b = Best{g_s[u], j_s[u], o_s[u] >> 1, (o_s[u] & 1) == 0 ? 1u : 0u, 1};
                }
            }
            uint32_t const side = (out->small_left != 0) != (lg != 0) ? 0 : 1;
            part[(side * gridDim.x) + blockIdx.x] = b;
            __threadfence();
        }
    }
    __syncthreads();
    if (threadIdx.x == 0)
    {
        __threadfence();
        last_s = atomicAdd(ticket, 1U) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last_s)
    {
        return;
    }
    __threadfence();
    if (work)
    {
        // a half of the CTA per child: the CTAs' choices, features in order
        uint32_t const x = threadIdx.x / (k_pop_thr / 2);
        double         g = 0.0;
        uint32_t       o = 0xFFFFFFFFu;
        for (uint32_t v = threadIdx.x % (k_pop_thr / 2); v < gridDim.x; v += k_pop_thr / 2)
        {
            Best const  *b  = part + (x * gridDim.x) + v;
            double const bg = __ldcg(&b->gain);
            if (__ldcg(&b->valid) != 0 && (bg > g || (bg == g && v < o)))
            {
                g = bg;
                o = v;
            }
        }
        warp_best(g, o);
        if (lane == 0)
        {
            g_s[w] = g;
            o_s[w] = o;
        }
        __syncthreads();
        if (threadIdx.x < 2)
        {
            uint32_t const w0 = threadIdx.x * (warps / 2);
            g                 = g_s[w0];
            o                 = o_s[w0];
            for (uint32_t v = w0 + 1; v < w0 + (warps / 2); ++v)
            {
                if (g_s[v] > g || (g_s[v] == g && o_s[v] < o))
                {
                    g = g_s[v];
                    o = o_s[v];
                }
            }
            Best b = {0.0, 0, 0, 1, 0};
            if (o != 0xFFFFFFFFu)
            {
                Best const *src = part + (threadIdx.x * gridDim.x) + o;
                b = Best{__ldcg(&src->gain), __ldcg(&src->feature), __ldcg(&src->bin),
                         __ldcg(&src->dl), __ldcg(&src->valid)};
            }
            out->best[threadIdx.x] = b;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        *ticket = 0; // ready for the next launch
    }
    leaf_turn(T, handle);
}

// The tree's epilogue: every remaining candidate is a leaf; the leaf list,
// node count and depth go to the level plane's control block.
__global__ void leaf_loop_end_kernel(LeafLoop *st, LeafCand const *cand, Node *leaves,
                                     Node *nodes, Ctl *ctl)
{
    pdl_enter();
    uint32_t const nl = st->n_leaves;
    uint32_t const nc = st->n_cand;
    for (uint32_t i = threadIdx.x; i < nl + nc; i += blockDim.x)
    {
        nodes[i] = i < nl ? leaves[i] : cand[i - nl].node;
    }
    if (threadIdx.x == 0)
    {
        ctl->n_cur    = nl + nc;
        ctl->n_nodes  = st->n_nodes;
        ctl->depth    = st->depth;
        ctl->n_leaves = 0;
    }
}

__global__ void leaf_set_tree_kernel(TreeOut *dst, TreeOut t, LeafLoop *st, uint32_t root_may)
{
    pdl_enter();
    *dst          = t;
    st->root_may  = root_may;
}

template <typename T> T *dalloc(size_t n, cudaStream_t s)
{
    void *p = nullptr;
    BB_CHECK(cudaMallocAsync(&p, std::max<size_t>(1, n) * sizeof(T), s));
    return static_cast<T *>(p);
}

} // namespace

Grower::Grower(Plane const &plane, GrowConfig const &cfg, std::vector<uint32_t> selected,
               uint32_t max_root_rows, cudaStream_t stream)
    : plane_(plane), cfg_(cfg), sel_h_(std::move(selected)), stream_(stream)
{
    if (cfg_.sample_k > 0)
    {
        // per-tree samples: the first sample_k features until set_selection
        if (cfg_.sample_k > plane_.n_feats || cfg_.sel_sets == 0)
        {
            throw ConfigError("grower: a feature sample larger than the plane");
        }
        sel_h_.resize(cfg_.sample_k);
        std::iota(sel_h_.begin(), sel_h_.end(), 0U);
    }
    n_sel_ = static_cast<uint32_t>(sel_h_.size());
    quant_ = cfg_.mode != HistMode::exact;
    pdl_   = quant_ && cfg_.lanes == 1;
    if (n_sel_ == 0)
    {
        throw ConfigError("grower: the feature selection is empty");
    }
    if (cfg_.leaf)
    {
        if (cfg_.tp.max_leaves == 0 && cfg_.tp.max_depth <= 9)
        {
            cfg_.tp.max_leaves = 1u << cfg_.tp.max_depth; // unbounded: the depth's cap
        }
        if (cfg_.tp.max_leaves < 1 || cfg_.tp.max_leaves > 512 || cfg_.tp.max_depth > 255)
        {
            throw ConfigError("grower: leafwise needs 1 <= max_leaves <= 512 and "
                              "max_depth <= 255");
        }
    }
    else if (cfg_.tp.max_depth > 8)
    {
        throw ConfigError("grower: max_depth above 8 exceeds the level plane's "
                          "512-node frontier; use a host grower");
    }
    {
        uint64_t const fit_rows = std::max<uint64_t>(cfg_.fit_rows, max_root_rows);
        wide_codes_ = cfg_.mode == HistMode::quant16;
        // int16 sums always outgrow a packed 32-bit half; int8 sums do once
        // 127 x rows reaches 2^31 (16,909,320 rows)
        cw_ = wide_codes_ || (cfg_.mode == HistMode::quant8 && fit_rows * 127ULL >= (1ULL << 31))
                  ? 2
                  : 1;
        // the leaf sums add at most one unit per row: 2^38 up to 2^24 rows,
        // then one bit less per doubling, so no sum leaves the int64 range
        uint32_t lg = 24;
        while (lg < 62 && (uint64_t{1} << lg) < fit_rows)
        {
            ++lg;
        }
        fix_unit_ = std::ldexp(1.0, 62 - static_cast<int>(lg));
    }
    std::vector<uint32_t> off(n_sel_ + 1, 0);
    std::vector<uint32_t> nb(n_sel_, 0);
    for (uint32_t j = 0; j < n_sel_; ++j)
    {
        uint32_t const f = sel_h_[j];
        nb[j]            = plane_.h_cut_off[f + 1] - plane_.h_cut_off[f];
        off[j + 1]       = off[j] + nb[j];
        max_nb_          = std::max(max_nb_, nb[j]);
    }
    if (max_nb_ > k_max_bins)
    {
        throw ConfigError("grower: a feature has more than 4096 bins; lower "
                          "bin_mapper.max_bin or use a host grower");
    }
    total_cells_ = off[n_sel_];
    off_h_       = off;
    if (cfg_.sample_k > 0)
    {
        // bounds over every sample: the largest feature's bins, and per node
        // the cells of the sample_k largest features (off_h_ is read at the
        // whole sample and at its first feature only)
        std::vector<uint32_t> all(plane_.n_feats);
        for (uint32_t f = 0; f < plane_.n_feats; ++f)
        {
            all[f]  = plane_.h_cut_off[f + 1] - plane_.h_cut_off[f];
            max_nb_ = std::max(max_nb_, all[f]);
        }
        std::sort(all.begin(), all.end(), std::greater<>());
        total_cells_ = std::accumulate(all.begin(), all.begin() + n_sel_, 0U);
        off_h_.assign(n_sel_ + 1, 0);
        off_h_[1]      = max_nb_;
        off_h_[n_sel_] = total_cells_;
        if (max_nb_ > k_max_bins)
        {
            throw ConfigError("grower: a feature has more than 4096 bins; lower "
                              "bin_mapper.max_bin or use a host grower");
        }
    }
    cell_stride_ = offset_stride(max_nb_);
    // leafwise: a pool slot per live leaf plus the one being built; a pop
    // consumes a heap entry (at most 2 per split + the root), two nodes each
    max_front_   = cfg_.leaf ? cfg_.tp.max_leaves + 1 : 1u << cfg_.tp.max_depth;
    max_nodes_   = cfg_.leaf ? 4 * cfg_.tp.max_leaves : (2u << cfg_.tp.max_depth) - 1;
    max_rows_    = std::max<uint32_t>(max_root_rows, 1);
    crows_       = quant_ ? k_qbuild_rows : k_build_rows;
    // the histogram grid: one CTA per SM for a large fit, one per 2,048-row
    // chunk of the root for a small one (us a round at 14,000 / 40,000 /
    // 200,000 rows x 28, depth 6: 240 / 243 / 256, against 272 / 268 / 274 with
    // one per four chunks; 64 fits of 1,000-200,000 rows in flight 236 ms
    // against 257 for 100 rounds); growers side by side share the SMs (seven
    // classes: 1.05 ms a round at 581,012 rows against 1.17 with a CTA per SM
    // each, 1.40 against 1.68 at 1,000,000)
    qctas_       = cfg_.hist_ctas > 0
                       ? std::min(cfg_.hist_ctas, 64u * k_qctas)
                       : std::max(1u, std::min(k_qctas / std::min(cfg_.lanes, k_qctas),
                                               ceil_div(max_rows_, k_qbuild_rows)));
    max_pchunks_ = ceil_div(max_rows_, k_part_rows) + max_front_;
    max_bchunks_ = ceil_div(max_rows_, crows_) + max_front_;

    cudaStream_t   s     = stream_;
    uint32_t const nsets = std::max(1u, cfg_.sel_sets);
    arena_.want<uint32_t>(sel_base_, static_cast<size_t>(nsets) * n_sel_);
    arena_.want<uint32_t>(cell_off_base_, static_cast<size_t>(nsets) * (n_sel_ + 1));
    arena_.want<uint32_t>(sel_nb_base_, static_cast<size_t>(nsets) * n_sel_);
    {
        // the mirror tiles a selection can touch: all selected features (v
        // 0), and the first one alone (v 1: the last level builds only its
        // totals); a sampled grower sizes them for any sample
        uint32_t const per     = k_mirror_bytes / (plane_.u8 ? 1 : 2);
        uint32_t const n_tiles = ceil_div(plane_.n_feats, per);
        for (int v = 0; v < 2; ++v)
        {
            uint32_t cap = 1;
            if (v == 0)
            {
                cap = 0;
                for (uint32_t j = 0; j < n_sel_; ++j)
                {
                    cap += (j == 0 || sel_h_[j] / per != sel_h_[j - 1] / per) ? 1 : 0;
                }
                if (cfg_.sample_k > 0)
                {
                    cap = std::min(n_sel_, n_tiles);
                }
            }
            n_tiles_[v]       = cap;
            arena_.want<uint32_t>(tile_ids_base_[v], static_cast<size_t>(nsets) * cap);
            arena_.want<int32_t>(tile_j_base_[v], static_cast<size_t>(nsets) * cap * per);
        }
    }
    arena_.want<Ctl>(ctl_, 1);
    arena_.want<Node>(nodes_[0], max_front_);
    arena_.want<Node>(nodes_[1], max_front_);
    arena_.want<float2>(hist_[0], static_cast<size_t>(max_front_) * total_cells_ * cw_);
    // (leafwise uses the first buffer as its slot pool)
    arena_.want<float2>(hist_[1],
                        static_cast<size_t>(cfg_.leaf ? 1 : max_front_) * total_cells_ * cw_);
    arena_.want<Best>(cand_, static_cast<size_t>(max_front_) * n_sel_);
    arena_.want<Best>(best_, max_front_);
    arena_.want<uint4>(route_, max_front_);
    arena_.want<Chunk>(pchunks_, max_pchunks_);
    arena_.want<uint32_t>(pleft_, max_pchunks_);
    arena_.want<uint32_t>(dirs_, static_cast<size_t>(max_pchunks_) * (k_part_rows / 32));
    arena_.want<uint32_t>(prbase_, max_pchunks_);
    arena_.want<uint32_t>(dst_, max_front_ + 1);
    arena_.want<uint32_t>(build_, max_front_ * 2 + 2);
    arena_.want<uint32_t>(bpair_, 3 * max_front_);
    arena_.want<uint32_t>(bbase_, max_front_ + 1);
    arena_.want<uint32_t>(brange_, max_front_ + 2);
    arena_.want<Chunk>(bchunks_, max_bchunks_);
    // (leafwise: two halves of one buffer, a node's segment in either, while a
    // 32-bit index reaches both; from 2^31 rows on a second buffer, whose rows
    // each pop copies back)
    bool const far = max_rows_ >= k_far_rows;
    arena_.want<uint32_t>(rows_[0], static_cast<size_t>(max_rows_) * (cfg_.leaf && !far ? 2 : 1));
    if (!cfg_.leaf || far)
    {
        arena_.want<uint32_t>(rows_[1], max_rows_);
    }
    arena_.want<uint32_t>(pcr_, max_front_ + 2);
    arena_.want<double2>(nbound_, std::max<uint32_t>(max_nodes_, k_walk_nodes));
    arena_.want<uint2>(heap_, k_heap_slots);
    arena_.want<uint16_t>(leafmap_, k_heap_slots + 1);
    if (cfg_.leaf)
    {
        arena_.want<LeafOut>(lout_, 1);
        arena_.want<uint32_t>(slot_of_, 2);
        arena_.want<LeafLoop>(loop_, 1);
        arena_.want<LeafCand>(cand_heap_, max_front_ + 2);
        arena_.want<Node>(leaves_, max_front_ + 2);
        arena_.want<uint32_t>(free_, max_front_ + 2);
        arena_.want<TreeOut>(tree_dev_, 1);
        arena_.want<uint32_t>(leaf_tick_, 2);
        BB_CHECK(cudaMallocHost(&lout_h_, sizeof(LeafLoop)));
    }
    arena_.want<uint32_t>(nleft_, max_front_ + 1);
    arena_.want<uint32_t>(nright_, max_front_ + 1);
    arena_.want<uint32_t>(dtree_, 1);
    if (quant_)
    {
        arena_.want<uint32_t>(absmax_, 2);
        arena_.want<double2>(qscale_, 1);
        // +2: the histogram copies whole 4-byte words of codes
        arena_.want<uint16_t>(qgh8_, (max_rows_ > plane_.n_rows ? max_rows_ : plane_.n_rows) + 2);
        if (wide_codes_)
        {
            arena_.want<uint32_t>(qgh16_, (max_rows_ > plane_.n_rows ? max_rows_ : plane_.n_rows) + 1);
        }
        arena_.want<double2>(partial_, max_pchunks_);
        arena_.want<int64_t>(btot_, 2 * static_cast<size_t>(max_front_));
        arena_.want<uint32_t>(done_, 1);
        arena_.want<unsigned long long>(wacc_, 2 * k_walk_nodes);
        arena_.want<uint16_t>(leaf16_, plane_.n_rows);
        uint32_t const per = k_mirror_bytes / (plane_.u8 ? 1 : 2);
        size_t const qsmem = static_cast<size_t>(per) * max_nb_ * 8;
        if (qsmem > 200 * 1024)
        {
            throw ConfigError("grower: quantised histograms of this many bins exceed "
                              "shared memory; lower bin_mapper.max_bin");
        }
        allow_smem(qhist_kernel<uint16_t>);
        allow_smem(qhist_kernel<uint16_t, true>);
        allow_smem(qhist_kernel<uint16_t, false, true>);
        allow_smem(qhist_kernel<uint8_t, true>);
        allow_smem(qhist_t_kernel<false>);
        allow_smem(qhist_t_kernel<true>);
        allow_smem(walk_sum_kernel<true, false>);
        allow_smem(walk_sum_kernel<true, true>);
        allow_smem(walk_sum_kernel<false, false>);
        allow_smem(walk_sum_kernel<false, true>);
    }
    else
    {
        arena_.want<uint16_t>(coff_, static_cast<size_t>(max_bchunks_) * n_sel_ * cell_stride_);
        // every built row once, and each chunk's padding
        p_stride_ = ((uint64_t{max_rows_} + 1) & ~uint64_t{1}) +
                    (uint64_t{max_bchunks_} * (chunk_pads(max_nb_) + 2));
        arena_.want<float2>(payload_, n_sel_ * p_stride_);
    }
    arena_.want<float2>(scale_, 1);
    arena_.want<uint32_t>(ticket_, max_front_ + 1);
    arena_.alloc(plane_.pool(), s);
    sets_h_.assign(nsets, sel_h_);
    for (uint32_t k = 0; k < nsets; ++k)
    {
        write_tables(k, sel_h_, s);
    }
    use_set(0);
    BB_CHECK(cudaMemsetAsync(scale_, 0, sizeof(float2), s));
    BB_CHECK(cudaMemsetAsync(dtree_, 0, 4, s));
    BB_CHECK(cudaMemsetAsync(ticket_, 0, (max_front_ + 1) * 4, s));
    if (cfg_.leaf)
    {
        BB_CHECK(cudaMemsetAsync(leaf_tick_, 0, 8, s));
    }
    if (quant_)
    {
        BB_CHECK(cudaMemsetAsync(done_, 0, 4, s));
    }
    BB_CHECK(cudaStreamSynchronize(s));

    // dynamic shared memory ceilings
    size_t const find_smem = max_nb_ * (sizeof(double2) + (sizeof(unsigned long long) * cw_));
    if (find_smem > 227 * 1024)
    {
        throw ConfigError("grower: bins per feature exceed the shared-memory budget");
    }
    allow_smem(find_kernel);
    // the level finder prefixes up to 16 nodes at a time in shared memory
    lgroup_ = static_cast<uint32_t>(std::min<size_t>(
        k_lfind_thr / 32, std::max<size_t>(1, (192 * 1024) / (max_nb_ * sizeof(double2)))));
    allow_smem(level_find_kernel<false>);
    allow_smem(level_find_kernel<true>);
    if (!quant_)
    {
        if (max_nb_ > k_exact_bins)
        {
            throw ConfigError("grower: bins per feature exceed the shared-memory budget");
        }
        // four features in flight, or two where a group's counters take more
        // (features of several thousand bins)
        xgroups_ = sort_smem(max_nb_, k_xgroups) <= 226 * 1024 ? k_xgroups : 2;
        allow_smem(sort_kernel<uint8_t, k_xgroups>);
        allow_smem(sort_kernel<uint16_t, k_xgroups>);
        allow_smem(sort_kernel<uint16_t, 2>);
    }
    BB_CHECK(cudaEventCreate(&pev_[0]));
    BB_CHECK(cudaEventCreate(&pev_[1]));
}

// Set k's tables for the ascending feature ids sel: the ids, each one's
// first cell and bin count, and the mirror tiles holding them
// with each tile slot's selection index, unused slots marked. The host
// vectors are pageable, so each copy has left them when it returns.
void Grower::write_tables(uint32_t set, std::vector<uint32_t> const &sel, cudaStream_t s)
{
    std::vector<uint32_t> off(n_sel_ + 1, 0);
    std::vector<uint32_t> nb(n_sel_, 0);
    for (uint32_t j = 0; j < n_sel_; ++j)
    {
        uint32_t const f = sel[j];
        nb[j]            = plane_.h_cut_off[f + 1] - plane_.h_cut_off[f];
        off[j + 1]       = off[j] + nb[j];
    }
    BB_CHECK(cudaMemcpyAsync(sel_base_ + (static_cast<size_t>(set) * n_sel_), sel.data(),
                             n_sel_ * 4, cudaMemcpyHostToDevice, s));
    BB_CHECK(cudaMemcpyAsync(cell_off_base_ + (static_cast<size_t>(set) * (n_sel_ + 1)),
                             off.data(), (n_sel_ + 1) * 4, cudaMemcpyHostToDevice, s));
    BB_CHECK(cudaMemcpyAsync(sel_nb_base_ + (static_cast<size_t>(set) * n_sel_), nb.data(),
                             n_sel_ * 4, cudaMemcpyHostToDevice, s));
    uint32_t const per = k_mirror_bytes / (plane_.u8 ? 1 : 2);
    for (int v = 0; v < 2; ++v)
    {
        uint32_t const        cap = n_tiles_[v];
        std::vector<uint32_t> ids;
        std::vector<int32_t>  js(static_cast<size_t>(cap) * per, -1);
        uint32_t const        nfb = v == 0 ? n_sel_ : 1;
        for (uint32_t j = 0; j < nfb; ++j)
        {
            uint32_t const t = sel[j] / per;
            if (ids.empty() || ids.back() != t)
            {
                ids.push_back(t);
            }
            js[((ids.size() - 1) * per) + (sel[j] % per)] = static_cast<int32_t>(j);
        }
        if (ids.size() > cap)
        {
            throw std::logic_error("grower: a selection touches more tiles than its tables hold");
        }
        ids.resize(cap, k_no_sel_tile);
        BB_CHECK(cudaMemcpyAsync(tile_ids_base_[v] + (static_cast<size_t>(set) * cap), ids.data(),
                                 cap * 4, cudaMemcpyHostToDevice, s));
        BB_CHECK(cudaMemcpyAsync(tile_j_base_[v] + (static_cast<size_t>(set) * cap * per),
                                 js.data(), js.size() * 4, cudaMemcpyHostToDevice, s));
    }
}

void Grower::set_selection(uint32_t set, std::vector<uint32_t> const &sel, cudaStream_t s)
{
    if (cfg_.sample_k == 0 || set >= sets_h_.size() || sel.size() != n_sel_)
    {
        throw std::logic_error("grower: set_selection outside a sampled grower's sets");
    }
    for (size_t j = 0; j < sel.size(); ++j)
    {
        if (sel[j] >= plane_.n_feats || (j > 0 && sel[j] <= sel[j - 1]))
        {
            throw std::logic_error("grower: a feature sample must be ascending plane features");
        }
    }
    write_tables(set, sel, s);
    sets_h_[set] = sel;
}

void Grower::use_set(uint32_t set)
{
    if (set >= sets_h_.size())
    {
        throw std::logic_error("grower: no such selection set");
    }
    uint32_t const per = k_mirror_bytes / (plane_.u8 ? 1 : 2);
    sel_      = sel_base_ + (static_cast<size_t>(set) * n_sel_);
    cell_off_ = cell_off_base_ + (static_cast<size_t>(set) * (n_sel_ + 1));
    sel_nb_   = sel_nb_base_ + (static_cast<size_t>(set) * n_sel_);
    for (int v = 0; v < 2; ++v)
    {
        if (tile_ids_base_[v] != nullptr)
        {
            tile_ids_[v] = tile_ids_base_[v] + (static_cast<size_t>(set) * n_tiles_[v]);
            tile_j_[v]   = tile_j_base_[v] + (static_cast<size_t>(set) * n_tiles_[v] * per);
        }
    }
    sel_h_ = sets_h_[set];
    set_   = set;
}

Grower::LoopGraph::~LoopGraph()
{
    if (x != nullptr)
    {
        cudaGraphExecDestroy(x);
    }
    if (g != nullptr)
    {
        cudaGraphDestroy(g);
    }
}

Grower::~Grower()
{
    for (void *p : {static_cast<void *>(mono_), static_cast<void *>(fgroups_),
                    static_cast<void *>(gleft_)})
    {
        if (p != nullptr)
        {
            cudaFreeAsync(p, stream_);
        }
    }
    arena_.release();
    loops_.clear();
    cudaStreamSynchronize(stream_);
    if (lout_h_ != nullptr)
    {
        cudaFreeHost(lout_h_);
    }
    cudaEventDestroy(pev_[0]);
    cudaEventDestroy(pev_[1]);
}

void Grower::phase_begin()
{
    if (prof_ != nullptr)
    {
        BB_CHECK(cudaEventRecord(pev_[0], stream_));
    }
}

void Grower::phase_end(double &acc)
{
    if (prof_ != nullptr)
    {
        float ms = 0.0F;
        BB_CHECK(cudaEventRecord(pev_[1], stream_));
        BB_CHECK(cudaEventSynchronize(pev_[1]));
        BB_CHECK(cudaEventElapsedTime(&ms, pev_[0], pev_[1]));
        acc += ms;
    }
}

void Grower::set_shard(Reducer *r, uint64_t row_offset, uint64_t total_rows)
{
    if (r != nullptr && !quant_)
    {
        throw ConfigError("grower: a sharded fit needs the quantised form (integer "
                          "histograms combine exactly; float cells would not)");
    }
    if (r != nullptr && total_rows > std::max<uint64_t>(cfg_.fit_rows, max_rows_))
    {
        throw ConfigError("grower: a shard's grower must be sized for the whole fit's rows "
                          "(GrowConfig::fit_rows)");
    }
    red_        = r;
    row_off_    = row_offset;
    total_rows_ = total_rows;
    if (r != nullptr)
    {
        // a shard's rounds put NCCL's kernels between this grower's: plain
        // stream order there
        pdl_ = false;
    }
    if (gleft_ == nullptr)
    {
        gleft_ = dalloc<uint64_t>(max_front_, stream_);
        BB_CHECK(cudaStreamSynchronize(stream_));
    }
}

void Grower::set_tree_numbers(uint32_t first, uint32_t step)
{
    tree_step_ = step;
    BB_CHECK(cudaMemcpyAsync(dtree_, &first, 4, cudaMemcpyHostToDevice, stream_));
    BB_CHECK(cudaStreamSynchronize(stream_));
}

size_t Grower::device_bytes(Plane const &plane, GrowConfig const &cfg,
                            std::vector<uint32_t> const &selected, uint32_t max_root_rows)
{
    size_t   cells  = 0;
    uint32_t max_nb = 0;
    for (uint32_t const f : selected)
    {
        uint32_t const nb = plane.h_cut_off[f + 1] - plane.h_cut_off[f];
        cells += nb;
        max_nb = std::max(max_nb, nb);
    }
    size_t const n     = max_root_rows;
    size_t const front = cfg.leaf ? cfg.tp.max_leaves + 1 : size_t{1} << cfg.tp.max_depth;
    size_t       bytes = (16 * n) + (front * ((2 * cells * 16) + (selected.size() * 32)));
    if (cfg.mode == HistMode::exact)
    {
        size_t const chunks = (n / k_build_rows) + front + 1;
        bytes += selected.size() * ((8 * (n + (chunks * (chunk_pads(max_nb) + 2)))) +
                                    (chunks * 2 * offset_stride(max_nb)));
    }
    return bytes;
}

void Grower::seed_absmax(float2 const *gh)
{
    if (!quant_)
    {
        return;
    }
    cudaStream_t   s    = stream_;
    uint32_t const n    = static_cast<uint32_t>(plane_.n_rows);
    uint32_t const grid = std::min<uint32_t>(ceil_div(std::max<uint32_t>(n, 1), k_threads),
                                             148u * 8u);
    BB_CHECK(cudaMemsetAsync(absmax_, 0, 8, s));
    launch_k(pdl_, absmax_kernel, grid, k_threads, 0, s, gh, n, absmax_);
    BB_LAUNCH("absmax_kernel");
}

void Grower::quantise(float2 const *gh, uint32_t n, bool have_absmax, OpenArgs const &open)
{
    cudaStream_t s = stream_;
    uint32_t const grid = std::min<uint32_t>(
        std::max<uint32_t>(ceil_div(std::max<uint32_t>(n, 1), k_threads),
                           ceil_div(open.n_zero, 4 * k_threads)),
        148u * 8u);
    if (!have_absmax)
    {
        BB_CHECK(cudaMemsetAsync(absmax_, 0, 8, s));
        launch_k(pdl_, absmax_kernel, grid, k_threads, 0, s, gh, n, absmax_);
        BB_LAUNCH("absmax_kernel");
        n_launch_ += 1;
    }
    if (red_ != nullptr)
    {
        red_->max_u32(absmax_, 2, s); // the fit's maxima: one scale for every shard
    }
    uint2 const key = make_uint2(static_cast<uint32_t>(seed_),
                                 static_cast<uint32_t>(seed_ >> 32));
    if (wide_codes_)
    {
        launch_k(pdl_, quantise_kernel<true>, grid, k_threads, 0, s, gh, n, absmax_, key, dtree_,
                 qgh16_, qscale_, row_off_, open);
    }
    else
    {
        launch_k(pdl_, quantise_kernel<false>, grid, k_threads, 0, s, gh, n, absmax_, key, dtree_,
                 qgh8_, qscale_, row_off_, open);
    }
    BB_LAUNCH("quantise_kernel");
    n_launch_ += 1;
}

void Grower::build(uint32_t const *rows, uint32_t nfb, int dst, bool zeroed, uint32_t n_nodes)
{
    cudaStream_t s = stream_;
    // the root's chunks, or those of n_nodes smaller children (each at most
    // half of its parent's rows)
    uint32_t const n_chunks =
        std::min(max_bchunks_, ceil_div(zeroed ? max_rows_ / 2 : max_rows_, crows_) + n_nodes);
    phase_begin();
    if (quant_)
    {
        int const v = nfb == n_sel_ ? 0 : 1;
        if (!zeroed && !chain_)
        {
            launch_k(pdl_, zero_build_kernel, max_front_, k_threads, 0, s, ctl_, build_,
                     static_cast<unsigned long long *>(hist_[dst]), total_cells_ * cw_,
                     off_h_[nfb] * cw_);
            BB_LAUNCH("zero_build_kernel");
            n_launch_ += 1;
        }
        uint32_t const per   = k_mirror_bytes / (plane_.u8 ? 1 : 2);
        size_t const   qsmem = static_cast<size_t>(per) * max_nb_ * 8;
        dim3 const     grid(max_bchunks_, n_tiles_[v]);
        if (wide_codes_)
        {
            // int16 codes: the per-chunk kernel with two-word cells
            if (plane_.u8)
            {
                launch_k(pdl_, qhist_kernel<uint8_t, true>, grid, k_qthreads, qsmem, s, ctl_,
                         bchunks_, build_, rows, static_cast<uint4 const *>(plane_.mirror),
                         plane_.n_rows, qgh16_, tile_ids_[v], tile_j_[v], sel_nb_, cell_off_,
                         max_nb_, static_cast<unsigned long long *>(hist_[dst]), total_cells_);
            }
            else
            {
                launch_k(pdl_, qhist_kernel<uint16_t, true>, grid, k_qthreads, qsmem, s, ctl_,
                         bchunks_, build_, rows, static_cast<uint4 const *>(plane_.mirror),
                         plane_.n_rows, qgh16_, tile_ids_[v], tile_j_[v], sel_nb_, cell_off_,
                         max_nb_, static_cast<unsigned long long *>(hist_[dst]), total_cells_);
            }
        }
        else if (plane_.u8)
        {
            size_t const tsmem = k_tsmem;
            // CTAs per tile: the caller's count, else one per SM for a plane of
            // one tile, and about two waves over all tiles for a wide plane (a
            // CTA zeroes and flushes a 64 KB table per node, so many tiles
            // want fewer, longer CTAs each)
            // (at least enough CTAs that no CTA's share of the chunks can
            // overflow its 32-bit shared words)
            uint32_t const ctas = std::max(
                ceil_div(max_bchunks_, k_tshare_chunks),
                cfg_.hist_ctas > 0
                    ? qctas_
                    : std::max(1u, std::min(qctas_, ceil_div(2 * k_qctas, n_tiles_[v]))));
            auto const kern = cw_ == 2 ? qhist_t_kernel<true> : qhist_t_kernel<false>;
            launch_k(pdl_, kern, dim3(ctas, n_tiles_[v]), k_tthreads, tsmem, s, ctl_, bchunks_,
                     build_, rows, static_cast<uint4 const *>(plane_.mirror), plane_.n_rows, qgh8_,
                     tile_ids_[v], tile_j_[v], sel_nb_, cell_off_, max_nb_,
                     static_cast<unsigned long long *>(hist_[dst]), total_cells_);
        }
        else
        {
            auto const kern =
                cw_ == 2 ? qhist_kernel<uint16_t, false, true> : qhist_kernel<uint16_t>;
            launch_k(pdl_, kern, grid, k_qthreads, qsmem, s, ctl_, bchunks_, build_, rows,
                     static_cast<uint4 const *>(plane_.mirror), plane_.n_rows, qgh8_, tile_ids_[v],
                     tile_j_[v], sel_nb_, cell_off_, max_nb_,
                     static_cast<unsigned long long *>(hist_[dst]), total_cells_);
        }
        BB_LAUNCH("qhist_kernel");
        n_launch_ += 1;
    }
    else
    {
        int const       v    = nfb == n_sel_ ? 0 : 1;
        uint32_t const *crow = rows != nullptr ? rows : root_rows_;
        // a small build's chunks leave SMs idle: a tile's features are then
        // split over several CTAs, each staging the chunk's rows, up to two CTAs
        // an SM (20,000 rows x 28: the root's sort 65.9 us in one part, 19.7 in seven; the
        // round 618 and 332, leafwise 2,797 and 1,629, 24 fits in flight 126 and
        // 94 ms for 50 rounds)
        uint32_t const per   = k_mirror_bytes / (plane_.u8 ? 1 : 2);
        uint32_t const parts = std::max(
            1u, std::min(ceil_div(nfb == 1 ? 1u : std::min(per, plane_.n_feats), xgroups_),
                         296u / (n_chunks * n_tiles_[v])));
        auto           sort = [&](auto kern)
        {
            launch_k(pdl_, kern, dim3(n_chunks, n_tiles_[v], parts), xgroups_ * k_xgthr,
                     sort_smem(max_nb_, xgroups_), s, ctl_, bchunks_, brange_, build_, crow,
                     static_cast<uint4 const *>(plane_.mirror), plane_.n_rows, gh_cur_,
                     tile_ids_[v], tile_j_[v], sel_nb_, cell_off_, max_nb_, nfb, coff_,
                     cell_stride_, payload_, p_stride_, static_cast<float2 *>(hist_[dst]),
                     total_cells_);
        };
        plane_.u8 ? sort(sort_kernel<uint8_t, k_xgroups>)
                  : (xgroups_ == 2 ? sort(sort_kernel<uint16_t, 2>)
                                   : sort(sort_kernel<uint16_t, k_xgroups>));
        BB_LAUNCH("sort_kernel");
        launch_k(pdl_, chain_kernel, dim3(n_nodes, nfb, ceil_div(max_nb_, 32)), k_cthreads, 0, s,
                 ctl_, build_, bchunks_, brange_, coff_, payload_, p_stride_, sel_nb_, cell_off_,
                 max_nb_, nfb, cell_stride_, static_cast<float2 *>(hist_[dst]), total_cells_);
        BB_LAUNCH("chain_kernel");
        n_launch_ += 2;
    }
    if (prof_ != nullptr)
    {
        double const before = prof_->hist_ms;
        phase_end(prof_->hist_ms);
        Ctl c{};
        BB_CHECK(cudaMemcpy(&c, ctl_, sizeof(Ctl), cudaMemcpyDeviceToHost));
        double const bin_bytes = plane_.u8 ? 1.0 : 2.0;
        // per built row: the codes read, the gradient pair, the row id
        double const per_row = quant_ ? ((nfb * bin_bytes) + 2.0 + 4.0)
                                      : ((nfb * bin_bytes) + 8.0 + 4.0);
        prof_->hist_rows += c.built_rows;
        prof_->hist_bytes += (static_cast<double>(c.built_rows) * per_row) +
                             (static_cast<double>(c.n_build) * off_h_[nfb] * 8.0);
        if (prof_->hist_builds < Profile::k_prof_builds)
        {
            prof_->build_ms[prof_->hist_builds]   = prof_->hist_ms - before;
            prof_->build_rows[prof_->hist_builds] = c.built_rows;
        }
        prof_->hist_builds += 1;
    }
}

void Grower::leaf_values(TreeOut const &t, bool)
{
    if (!quant_)
    {
        return;
    }
    cudaStream_t s = stream_;
    launch_k(pdl_, leafsum_kernel, max_pchunks_, k_threads, 0, s, ctl_, pchunks_, nodes_cur_,
             rows_cur_, gh_cur_, partial_, pcr_, cfg_.tp, t, done_);
    BB_LAUNCH("leafsum_kernel");
    n_launch_ += 1;
}

void Grower::level(uint32_t L, uint32_t const *rows_in, uint32_t *rows_out,
                   TreeOut const &t, uint32_t *leaf_id, float *scores, float lr)
{
    cudaStream_t s   = stream_;
    int const    cur = static_cast<int>(L & 1);
    int const    nxt = cur ^ 1;
    // grids sized for this level: at most 2^L frontier nodes, and at most one
    // partial partition chunk per node beyond the rows' whole chunks
    uint32_t const front = std::min(max_front_, 1u << std::min(L, 30u));
    uint32_t const pch   = std::min(max_pchunks_, ceil_div(max_rows_, k_part_rows) + front);
    size_t const find_smem = max_nb_ * (sizeof(double2) + (sizeof(unsigned long long) * cw_));
    phase_begin();
    dim3 const fgrid(front, n_sel_);
    HeapOut const ho{heap_, leafmap_, cfg_.tp.max_depth, k_mirror_bytes / (plane_.u8 ? 1u : 2u)};
    PlanArgs const plan{sel_, plane_.cuts, plane_.cut_off, cfg_.tp, t,      pchunks_,
                        pcr_, nbound_,     ho,             nleft_,  nright_, route_};
    FindChain const chain{ctl_,
                          nodes_[cur],
                          best_,
                          btot_,
                          ticket_,
                          static_cast<unsigned long long *>(hist_[cur]),
                          L > 0 ? static_cast<unsigned long long const *>(hist_[nxt]) : nullptr,
                          bpair_,
                          plan};
    if (cfg_.level)
    {
        size_t const lsmem = static_cast<size_t>(lgroup_) * max_nb_ * sizeof(double2);
        auto const   kern  = quant_ ? level_find_kernel<true> : level_find_kernel<false>;
        launch_k(pdl_, kern, n_sel_, k_lfind_thr, lsmem, s, ctl_, nodes_[cur], hist_[cur],
                 total_cells_, cell_off_, sel_nb_, n_sel_, cfg_.tp, cand_, max_nb_, lgroup_,
                 qscale_, cw_);
    }
    else if (quant_)
    {
        auto const kern = packed_  ? qfind_warp_kernel<false, true>
                          : cw_ == 2 ? qfind_warp_kernel<true, false>
                                     : qfind_warp_kernel<false, false>;
        launch_k(pdl_, kern, dim3(front, ceil_div(n_sel_, k_qfind_warps)), k_qfind_warps * 32, 0, s,
                 ctl_, nodes_[cur], hist_[cur], total_cells_, cell_off_, sel_nb_, sel_, n_sel_,
                 mono_, n_mono_, cfg_.tp, cand_, qscale_, fgroups_, chain);
    }
    else
    {
        launch_k(pdl_, find_kernel, fgrid, k_find_thr, find_smem, s, ctl_, nodes_[cur],
                 hist_[cur], total_cells_, cell_off_, sel_nb_, sel_, n_sel_, mono_, n_mono_,
                 cfg_.tp, cand_, max_nb_, nullptr, fgroups_);
    }
    BB_LAUNCH("find_kernel");
    if (!packed_)
    {
        launch_k(pdl_, plan_kernel, 1, k_plan_thr, 0, s, ctl_, nodes_[cur], cand_, best_, n_sel_,
                 cfg_.level, plan);
        BB_LAUNCH("plan_kernel");
    }
    if (prof_ != nullptr)
    {
        phase_end(prof_->find_ms);
    }
    phase_begin();
    bool const     last     = (L + 1) == cfg_.tp.max_depth;
    uint32_t const nfb      = last ? 1 : n_sel_;
    uint32_t const n_zcells = quant_ && !last ? off_h_[nfb] * cw_ : 0;
    Plan2Args const plan2{ctl_,   nodes_[cur], nodes_[nxt], best_,   pchunks_, pcr_,
                          pleft_, prbase_,     nleft_,      dst_,    bpair_,   build_,
                          brange_, bchunks_,   cfg_.tp,     t,       crows_,   bbase_,
                          cfg_.level, red_ != nullptr ? gleft_ : nullptr, fgroups_, ho,
                          packed_ ? btot_ : nullptr, sel_, mono_, n_mono_, qscale_,
                          packed_ && last, nbound_, dtree_, tree_step_};
    // a walked quantised tree (unsharded) partitions in one pass: nothing
    // downstream of its row lists depends on the rows' order inside a node
    if (chain_)
    {
        auto const kern = plane_.u8 ? (last ? psplit_kernel<uint8_t, false>
                                            : psplit_kernel<uint8_t, true>)
                                    : (last ? psplit_kernel<uint16_t, false>
                                            : psplit_kernel<uint16_t, true>);
        launch_k(pdl_, kern, pch, k_threads, 0, s, ctl_, pchunks_, nodes_[cur], route_,
                 rows_in, rows_out, plane_.bins, plane_.n_pad, nleft_, nright_,
                 static_cast<unsigned long long *>(hist_[nxt]), total_cells_ * cw_, n_zcells);
        BB_LAUNCH("psplit_kernel");
    }
    else if (plane_.u8)
    {
        launch_k(pdl_, pcount_kernel<uint8_t, false>, pch, k_threads, 0, s, ctl_, pchunks_,
                 nodes_[cur], best_, rows_in, plane_.bins, plane_.n_pad, sel_, sel_nb_, pleft_,
                 dirs_, LeafPlanArgs{});
    }
    else
    {
        launch_k(pdl_, pcount_kernel<uint16_t, false>, pch, k_threads, 0, s, ctl_, pchunks_,
                 nodes_[cur], best_, rows_in, plane_.bins, plane_.n_pad, sel_, sel_nb_, pleft_,
                 dirs_, LeafPlanArgs{});
    }
    BB_LAUNCH("partition kernel");
    if (red_ != nullptr)
    {
        launch_k(pdl_, node_left_kernel, 1, k_plan_thr, 0, s, ctl_, pcr_, pleft_, gleft_,
                 max_front_);
        BB_LAUNCH("node_left_kernel");
        red_->sum_u64(gleft_, max_front_, s);
        n_launch_ += 1;
    }
    launch_k(pdl_, chain_ ? plan2_kernel<true> : plan2_kernel<false>, 1, k_plan_thr, 0, s, plan2);
    BB_LAUNCH("plan2_kernel");
    nodes_cur_ = nodes_[cur];
    rows_cur_  = rows_in;
    if (!(walk_ && quant_))
    {
        leaf_values(t, false);
    }
    if (!walk_)
    {
        launch_k(pdl_, stamp_kernel, pch, k_threads, 0, s, ctl_, pchunks_, nodes_[cur],
                 rows_in, t, leaf_id, scores, lr);
        BB_LAUNCH("stamp_kernel");
        n_launch_ += 1;
    }
    if (packed_)
    {
        if (prof_ != nullptr)
        {
            phase_end(prof_->partition_ms);
        }
        n_launch_ += 3;
        if (!last)
        {
            build(rows_out, nfb, nxt, true, front);
        }
        return;
    }
    if (quant_ && last && walk_)
    {
        // a walked tree's last level: the leaves' rows are never listed (the
        // walk routes every row) and their exact totals come from the
        // parents' split cells
        if (prof_ != nullptr)
        {
            phase_end(prof_->partition_ms);
        }
        phase_begin();
        launch_k(pdl_, qsplit_totals_kernel, ceil_div(std::min(max_front_, 2 * front), 8u), 256, 0, s, ctl_, bpair_,
                 nodes_[cur], best_, static_cast<unsigned long long const *>(hist_[cur]),
                 total_cells_, cell_off_, sel_nb_, cw_, btot_);
        BB_LAUNCH("qsplit_totals_kernel");
        launch_k(pdl_, qsubtract_totals_kernel, front, k_threads, 0, s, ctl_, bpair_,
                 static_cast<unsigned long long const *>(hist_[cur]),
                 static_cast<unsigned long long *>(hist_[nxt]), total_cells_, 0, nodes_[cur],
                 nodes_[nxt], best_, sel_, sel_nb_, mono_, n_mono_, cfg_.tp, qscale_, btot_, cw_);
        BB_LAUNCH("qsubtract_totals_kernel");
        n_launch_ += 6; // count, plan2, the two totals kernels (+ find, plan)
        if (prof_ != nullptr)
        {
            phase_end(prof_->other_ms);
        }
        return;
    }
    if (!chain_)
    {
        launch_k(pdl_, pscatter_kernel, pch, k_threads, 0, s, ctl_, pchunks_, nodes_[cur], best_,
                 pleft_, prbase_, nleft_, dst_, rows_in, rows_out, dirs_,
                 static_cast<unsigned long long *>(hist_[nxt]), build_, total_cells_ * cw_,
                 n_zcells);
        BB_LAUNCH("pscatter_kernel");
    }
    if (prof_ != nullptr)
    {
        phase_end(prof_->partition_ms);
    }
    n_launch_ += chain_ ? 4 : 5;
    if (quant_ && last)
    {
        // the last level's nodes are leaves: the quantised form needs their
        // exact totals only (monotone bounds), not their histograms
        phase_begin();
        BB_CHECK(cudaMemsetAsync(btot_, 0, sizeof(int64_t) * 2 * max_front_, s));
        launch_k(pdl_, qbuilt_totals_kernel, max_bchunks_, k_threads, 0, s, ctl_, bchunks_,
                 rows_out, qgh8_, qgh16_, btot_);
        BB_LAUNCH("qbuilt_totals_kernel");
        if (red_ != nullptr)
        {
            red_->sum_u64(btot_, 2 * static_cast<size_t>(max_front_), s);
        }
        launch_k(pdl_, qsubtract_totals_kernel, front, k_threads, 0, s, ctl_, bpair_,
                 static_cast<unsigned long long const *>(hist_[cur]),
                 static_cast<unsigned long long *>(hist_[nxt]), total_cells_, 0, nodes_[cur],
                 nodes_[nxt], best_, sel_, sel_nb_, mono_, n_mono_, cfg_.tp, qscale_, btot_, cw_);
        BB_LAUNCH("qsubtract_totals_kernel");
        n_launch_ += 2;
        if (prof_ != nullptr)
        {
            phase_end(prof_->other_ms);
        }
        return;
    }
    build(rows_out, nfb, nxt, true, front);
    uint32_t const n_cells = off_h_[nfb]; // the built features: a selection prefix
    if (red_ != nullptr)
    {
        // the next frontier's slots (at most 2^(L+1)): the built ones carry
        // this shard's partial cells, the rest are rewritten by the subtraction
        size_t const slots = std::min<size_t>(size_t{2} << L, max_front_);
        red_->sum_u64(hist_[nxt], slots * total_cells_ * cw_, s);
    }
    phase_begin();
    if (quant_)
    {
        launch_k(pdl_, qsubtract_totals_kernel,
                 dim3(front, std::max(1u, ceil_div(n_cells * cw_, k_sub_cells))), k_threads, 0,
                 s, ctl_, bpair_, static_cast<unsigned long long const *>(hist_[cur]),
                 static_cast<unsigned long long *>(hist_[nxt]), total_cells_, n_cells, nodes_[cur],
                 nodes_[nxt], best_, sel_, sel_nb_, mono_, n_mono_, cfg_.tp, qscale_, nullptr, cw_);
        BB_LAUNCH("qsubtract_totals_kernel");
    }
    else
    {
        launch_k(pdl_, subtract_totals_kernel,
                 dim3(front, std::max(1u, ceil_div(n_cells, k_sub_cells))), k_threads, 0, s, ctl_,
                 bpair_,
                 static_cast<float2 const *>(hist_[cur]), static_cast<float2 *>(hist_[nxt]),
                 total_cells_, n_cells, nodes_[cur], nodes_[nxt], best_, sel_, sel_nb_, mono_,
                 n_mono_, cfg_.tp);
        BB_LAUNCH("subtract_totals_kernel");
    }
    n_launch_ += 1;
    if (prof_ != nullptr)
    {
        phase_end(prof_->other_ms);
    }
}

void Grower::grow(float2 const *gh, uint32_t const *root_rows, uint32_t n_root,
                  TreeOut const &t, uint32_t *leaf_id, float *scores, float lr,
                  bool identity_root, NextRound const *next, RootSample const *sample,
                  TreeCommit const &commit)
{
    if (n_root > max_rows_)
    {
        throw ConfigError("grower: more sampled rows than the grower was sized for");
    }
    cudaStream_t s = stream_;
    gh_cur_        = gh;
    root_rows_     = root_rows;
    n_launch_      = 0;
    if (cfg_.leaf)
    {
        if (next != nullptr || red_ != nullptr || sample != nullptr)
        {
            throw ConfigError("grower: the leafwise plane takes neither a fused next round "
                              "nor row shards");
        }
        walk_ = false;
        if (quant_)
        {
            quantise(gh, static_cast<uint32_t>(plane_.n_rows), false, OpenArgs{});
        }
        grow_leafwise(root_rows, n_root, t, leaf_id, scores, lr);
        return;
    }
    if (sample != nullptr && (identity_root || red_ != nullptr))
    {
        throw ConfigError("grower: a device row sample is neither the identity root nor a "
                          "row shard");
    }
    walk_ = (sample != nullptr || (identity_root && n_root == plane_.n_rows)) &&
            (leaf_id != nullptr || scores != nullptr || next != nullptr);
    if (next != nullptr && !walk_)
    {
        throw ConfigError("grower: a fused next round needs every row as the root");
    }
    if (red_ != nullptr && (!quant_ || !walk_))
    {
        throw ConfigError("grower: a sharded fit needs the quantised form and every row as "
                          "the root");
    }
    // (a shard's cells are the fit's only after a reduction between launches)
    chain_  = quant_ && walk_ && red_ == nullptr;
    packed_ = chain_ && !cfg_.level && cw_ == 1 && cfg_.tp.max_depth > 0;
    uint32_t const g_root = red_ != nullptr ? static_cast<uint32_t>(total_rows_) : n_root;
    RootArgs const root{ctl_, nodes_[0], n_root, bchunks_, brange_, build_, t, crows_, g_root,
                        sample != nullptr ? sample->count : nullptr, heap_};
    if (quant_)
    {
        phase_begin();
        OpenArgs open{};
        if (chain_)
        {
            open = OpenArgs{static_cast<unsigned long long *>(hist_[0]),
                            uint64_t{off_h_[cfg_.tp.max_depth == 0 ? 1 : n_sel_]} * cw_, wacc_, root};
        }
        quantise(gh, static_cast<uint32_t>(plane_.n_rows), next != nullptr, open);
        if (prof_ != nullptr)
        {
            phase_end(prof_->other_ms);
        }
    }
    if (!chain_)
    {
        launch_k(pdl_, root_setup_kernel, 1, k_threads, 0, s, root);
        BB_LAUNCH("root_setup_kernel");
        n_launch_ += 1;
    }
    // the root's rows: the quantised build reads an identity list implicitly
    build(quant_ && identity_root ? nullptr : root_rows,
          cfg_.tp.max_depth == 0 ? 1 : n_sel_, 0, false, 1);
    if (red_ != nullptr)
    {
        red_->sum_u64(hist_[0], total_cells_ * cw_, s);
    }
    phase_begin();
    if (!packed_)
    {
        if (quant_)
        {
            launch_k(pdl_, qroot_totals_kernel, 1, 32, 0, s, nodes_[0],
                     static_cast<unsigned long long const *>(hist_[0]), sel_nb_, cw_);
            BB_LAUNCH("qroot_totals_kernel");
        }
        else
        {
            launch_k(pdl_, root_totals_kernel, 1, 32, 0, s, nodes_[0],
                     static_cast<float2 const *>(hist_[0]), sel_nb_);
            BB_LAUNCH("root_totals_kernel");
        }
        n_launch_ += 1;
    }
    if (prof_ != nullptr)
    {
        phase_end(prof_->other_ms);
    }
    uint32_t const *rows_in = chain_ && identity_root ? nullptr : root_rows;
    for (uint32_t L = 0; L < cfg_.tp.max_depth; ++L)
    {
        uint32_t *rows_out = rows_[L & 1];
        level(L, rows_in, rows_out, t, leaf_id, scores, lr);
        rows_in = rows_out;
    }
    phase_begin();
    int const fin = static_cast<int>(cfg_.tp.max_depth & 1);
    if (!packed_)
    {
        launch_k(pdl_, final_kernel, 1, k_plan_thr, 0, s, ctl_, nodes_[fin], cfg_.tp, t, pchunks_,
                 pcr_, nbound_,
                 HeapOut{heap_, leafmap_, cfg_.tp.max_depth,
                         k_mirror_bytes / (plane_.u8 ? 1u : 2u)},
                 dtree_, tree_step_);
        BB_LAUNCH("final_kernel");
        n_launch_ += 1;
    }
    nodes_cur_ = nodes_[fin];
    rows_cur_  = rows_in;
    if (walk_)
    {
        uint32_t const n    = static_cast<uint32_t>(plane_.n_rows);
        uint32_t const grid = std::min<uint32_t>(ceil_div(std::max<uint32_t>(n, 1), k_threads),
                                                 148u * 8u);
        uint32_t const per   = k_mirror_bytes / (plane_.u8 ? 1u : 2u);
        bool const     multi = plane_.n_feats > per;
        auto const    *mir   = static_cast<uint4 const *>(plane_.mirror);
        uint32_t const depth = cfg_.tp.max_depth;
        WalkArgs a{};
        a.commit    = commit;
        a.scores    = scores;
        a.leaf_id   = leaf_id;
        a.lr        = lr;
        a.objective = next != nullptr ? next->objective : 0;
        a.weights   = next != nullptr ? next->weights : nullptr;
        a.labels    = next != nullptr ? next->labels : nullptr;
        a.gh        = next != nullptr ? next->gh : nullptr;
        a.absmax    = next != nullptr && quant_ ? absmax_ : nullptr;
        if (quant_)
        {
            if (!chain_)
            {
                BB_CHECK(cudaMemsetAsync(wacc_, 0, sizeof(unsigned long long) * 2 * k_walk_nodes,
                                         s));
            }
            FixArgs const fix{ctl_,    t,         wacc_, nbound_, absmax_, cfg_.tp, fix_unit_,
                              chain_ ? ticket_ : nullptr, next != nullptr ? absmax_ : nullptr};
            auto sum = [&](auto kern)
            {
                uint32_t const wgrid =
                    std::min<uint32_t>(ceil_div(std::max<uint32_t>(n, 1), k_wsum_thr), 148u * 2u);
                launch_k(pdl_, kern, wgrid, k_wsum_thr,
                         (size_t{2} << depth) * k_wsum_copies * sizeof(unsigned long long), s,
                         ctl_, mir, plane_.n_rows, heap_, leafmap_, depth, gh_cur_, absmax_,
                         leaf16_, wacc_, sample != nullptr ? sample->bits : nullptr, fix_unit_, fix);
            };
            if (plane_.u8)
            {
                multi ? sum(walk_sum_kernel<true, true>) : sum(walk_sum_kernel<true, false>);
            }
            else
            {
                multi ? sum(walk_sum_kernel<false, true>) : sum(walk_sum_kernel<false, false>);
            }
            BB_LAUNCH("walk_sum_kernel");
            if (red_ != nullptr)
            {
                red_->sum_u64(wacc_, 2 * static_cast<size_t>(k_walk_nodes), s);
            }
            if (!chain_)
            {
                launch_k(pdl_, leaf_fix_kernel, 1, k_threads, 0, s, fix);
                BB_LAUNCH("leaf_fix_kernel");
                n_launch_ += 1;
                if (next != nullptr)
                {
                    BB_CHECK(cudaMemsetAsync(absmax_, 0, 8, s));
                }
            }
            launch_k(pdl_, walk_apply_kernel, grid, k_threads, 0, s, ctl_, t, plane_.n_rows,
                     leaf16_, a);
            BB_LAUNCH("walk_apply_kernel");
            n_launch_ += 2;
        }
        else
        {
            auto walk = [&](auto kern)
            {
                launch_k(pdl_, kern, grid, k_threads, 0, s, ctl_, t, mir, plane_.n_rows, heap_,
                         leafmap_, depth, a);
            };
            if (plane_.u8)
            {
                multi ? walk(walk_kernel<true, true>) : walk(walk_kernel<true, false>);
            }
            else
            {
                multi ? walk(walk_kernel<false, true>) : walk(walk_kernel<false, false>);
            }
            BB_LAUNCH("walk_kernel");
            n_launch_ += 1;
        }
    }
    else
    {
        leaf_values(t, true);
        launch_k(pdl_, stamp_kernel, max_pchunks_, k_threads, 0, s, ctl_, pchunks_, nodes_[fin],
                 rows_in, t, leaf_id, scores, lr);
        BB_LAUNCH("stamp_kernel");
        n_launch_ += 1;
    }
    if (prof_ != nullptr)
    {
        phase_end(prof_->other_ms);
    }
    launches_ = n_launch_;
    ++tree_no_;
}

// LeafwiseGrower::grow on the device: the same gain heap (max gain, the lower
// node id on a tie), child ids allocated at the pop, demotion when the
// partition empties a side (its two children stay as zero leaf placeholders),
// no children's split at the depth cap, the leaf budget; the host launches the
// loop once and reads its verdict after the tree.
void Grower::grow_leafwise(uint32_t const *root_rows, uint32_t n_root, TreeOut const &t,
                           uint32_t *leaf_id, float *scores, float lr)
{
    cudaStream_t      s         = stream_;
    TreeParams const &tp        = cfg_.tp;
    size_t const      find_smem = max_nb_ * (sizeof(double2) + (sizeof(unsigned long long) * cw_));
    auto             *lout      = static_cast<LeafOut *>(lout_);
    auto             *st        = static_cast<LeafLoop *>(loop_);
    auto             *cand      = static_cast<LeafCand *>(cand_heap_);
    auto             *tdev      = static_cast<TreeOut *>(tree_dev_);
    LeafPop const    *pp        = &st->pop;
    bool const        far       = max_rows_ >= k_far_rows;
    void             *pool      = hist_[0];
    uint32_t          launches  = 0;
    LeafTurn const    turn{st,       cand,           leaves_,          free_,    lout,
                        tdev,     plane_.cuts,    plane_.cut_off,   sel_,     tp.max_leaves,
                        max_nodes_, tp.max_depth, 4 * max_front_ + 8, ctl_,   nodes_[0],
                        best_,    pchunks_,       pcr_};
    BB_CHECK(cudaMemcpyAsync(rows_[0], root_rows, size_t{n_root} * 4, cudaMemcpyDeviceToDevice,
                             s));
    launch_k(pdl_, leaf_set_tree_kernel, 1, 1, 0, s, tdev, t, st, tp.max_depth > 0 ? 1u : 0u);
    BB_LAUNCH("leaf_set_tree_kernel");
    launch_k(pdl_, root_setup_kernel, 1, k_threads, 0, s,
             RootArgs{ctl_, nodes_[0], n_root, bchunks_, brange_, build_, t, crows_, n_root, nullptr, nullptr});
    BB_LAUNCH("root_setup_kernel");
    launches += 2;
    build(rows_[0], n_sel_, 0, false, 1);
    if (quant_)
    {
        launch_k(pdl_, qroot_totals_kernel, 1, 32, 0, s, nodes_[0],
                 static_cast<unsigned long long const *>(pool), sel_nb_, cw_);
    }
    else
    {
        launch_k(pdl_, root_totals_kernel, 1, 32, 0, s, nodes_[0],
                 static_cast<float2 const *>(pool), sel_nb_);
    }
    BB_LAUNCH("root_totals_kernel");
    launches += 1;
    // each node's best split, then the pair's outcome (the children and their
    // bests) into lout; may_split: the depth cap's verdict, on the device
    auto find = [&](Node const *nodes, uint32_t const *slot_of, uint32_t const *may_split)
    {
        dim3 const fgrid(2, n_sel_);
        if (quant_)
        {
            // (the root's only: the pairs are found by leaf_pair_kernel)
            launch_k(pdl_, cw_ == 2 ? qfind_warp_kernel<true, false> : qfind_warp_kernel<false, false>,
                     dim3(2, ceil_div(n_sel_, k_qfind_warps)), k_qfind_warps * 32, 0, s, ctl_,
                     nodes, pool, total_cells_, cell_off_, sel_nb_, sel_, n_sel_, mono_, n_mono_,
                     tp, cand_, qscale_, fgroups_, FindChain{});
        }
        else
        {
            launch_k(pdl_, find_kernel, fgrid, k_find_thr, find_smem, s, ctl_, nodes, pool,
                     total_cells_, cell_off_, sel_nb_, sel_, n_sel_, mono_, n_mono_, tp, cand_,
                     max_nb_, slot_of, fgroups_);
        }
        BB_LAUNCH("find_kernel");
        launch_k(pdl_, leaf_best_kernel, 2, k_best_thr, 0, s, ctl_, cand_, n_sel_, nodes, lout,
                 may_split);
        BB_LAUNCH("leaf_best_kernel");
    };
    find(nodes_[0], nullptr, &st->root_may);
    launch_k(pdl_, leaf_loop_init_kernel, 1, k_plan_thr, 0, s, st, cand, leaves_, free_, lout, tdev,
             n_root, max_front_, tp.max_depth);
    BB_LAUNCH("leaf_loop_init_kernel");
    launch_k(pdl_, leaf_first_pop_kernel, 1, k_pop_thr, 0, s, turn);
    BB_LAUNCH("leaf_first_pop_kernel");
    launches += 4;

    // one pop as a fixed sequence of launches, repeated by the loop graph's
    // WHILE node until a turn (leaf_turn) finds nothing to pop; captured
    // once for these gradients and this table set (the loop's other buffers and
    // the tree's device record do not move)
    float2 const *const lgh  = quant_ ? nullptr : gh_cur_; // (the codes have one place)
    LoopGraph const    *loop = nullptr;
    for (auto const &l : loops_)
    {
        if (l->gh == lgh && l->set == set_)
        {
            loop = l.get();
        }
    }
    if (loop == nullptr)
    {
        Profile *const saved = prof_;
        prof_                = nullptr; // no per-phase events inside the loop graph
        auto made            = std::make_unique<LoopGraph>();
        made->gh             = lgh;
        made->set            = set_;
        BB_CHECK(cudaGraphCreate(&made->g, 0));
        cudaGraphConditionalHandle handle{};
        BB_CHECK(cudaGraphConditionalHandleCreate(&handle, made->g, 1,
                                                  cudaGraphCondAssignDefault));
        cudaGraphNodeParams cp{};
        cp.type               = cudaGraphNodeTypeConditional;
        cp.conditional.handle = handle;
        cp.conditional.type   = cudaGraphCondTypeWhile;
        cp.conditional.size   = 1;
        cudaGraphNode_t cnode{};
        BB_CHECK(cudaGraphAddNode(&cnode, made->g, nullptr, 0, &cp));
        cudaGraph_t const body = cp.conditional.phGraph_out[0];
        BB_CHECK(cudaStreamBeginCaptureToGraph(s, body, nullptr, nullptr, 0,
                                               cudaStreamCaptureModeThreadLocal));
        uint32_t const n0 = n_launch_;
        try
        {
            LeafPlanArgs const lp{ctl_,   pchunks_, pleft_, prbase_,   nleft_,     dst_,
                                  build_, brange_,  bbase_, bchunks_,  bpair_,     nodes_[0],
                                  nodes_[1], slot_of_, lout, crows_,   far ? 0u : max_rows_,
                                  pp,     leaf_tick_};
            auto count = [&](auto kern)
            {
                launch_k(pdl_, kern, max_pchunks_, k_threads, 0, s, ctl_, pchunks_, nodes_[0],
                         best_, rows_[0], plane_.bins, plane_.n_pad, sel_, sel_nb_, pleft_, dirs_,
                         lp);
            };
            plane_.u8 ? count(pcount_kernel<uint8_t, true>) : count(pcount_kernel<uint16_t, true>);
            BB_LAUNCH("pcount_kernel");
            launch_k(pdl_, pscatter_kernel, max_pchunks_, k_threads, 0, s, ctl_, pchunks_,
                     nodes_[0], best_, pleft_, prbase_, nleft_, dst_, rows_[0], rows_[far ? 1 : 0],
                     dirs_, static_cast<unsigned long long *>(pool), build_, total_cells_ * cw_,
                     quant_ ? total_cells_ * cw_ : 0);
            BB_LAUNCH("pscatter_kernel");
            n_launch_ = 2; // the body's so far: count, scatter
            if (far)
            {
                launch_k(pdl_, leaf_copyback_kernel, 148 * 4, k_threads, 0, s, pp, lout, rows_[1],
                         rows_[0]);
                BB_LAUNCH("leaf_copyback_kernel");
                n_launch_ += 1;
            }
            build(rows_[0], n_sel_, 0, true, 1);
            if (quant_)
            {
                launch_k(pdl_, cw_ == 2 ? leaf_pair_kernel<true> : leaf_pair_kernel<false>,
                         ceil_div(n_sel_, k_pop_thr / 64), k_pop_thr, 0, s, turn, lout, nodes_[1],
                         static_cast<unsigned long long *>(pool), total_cells_, cell_off_, sel_nb_,
                         n_sel_, mono_, n_mono_, tp, qscale_, fgroups_, cand_, leaf_tick_ + 1,
                         handle);
                BB_LAUNCH("leaf_pair_kernel");
                n_launch_ += 1;
            }
            else
            {
                uint32_t const sgrid =
                    std::max(1u, std::min(ceil_div(total_cells_, 256), 148u * 8u));
                auto *fpool = static_cast<float2 *>(pool);
                launch_k(pdl_, leaf_sub_kernel, sgrid, 256, 0, s, lout, bpair_, fpool,
                         total_cells_, total_cells_);
                BB_LAUNCH("leaf_sub_kernel");
                launch_k(pdl_, leaf_totals_kernel, 1, 64, 0, s, ctl_, lout, nodes_[1], slot_of_,
                         fpool, total_cells_, sel_, sel_nb_, mono_, n_mono_, tp, pp, fgroups_);
                BB_LAUNCH("leaf_totals_kernel");
                find(nodes_[1], slot_of_, &st->may_split);
                launch_k(pdl_, leaf_turn_kernel, 1, k_pop_thr, 0, s, turn, handle);
                BB_LAUNCH("leaf_turn_kernel");
                n_launch_ += 5; // subtraction, totals, find, best, turn
            }
            body_launches_ = n_launch_;
        }
        catch (...)
        {
            cudaGraph_t dummy{};
            cudaStreamEndCapture(s, &dummy);
            prof_     = saved;
            n_launch_ = n0;
            throw;
        }
        cudaGraph_t captured{};
        BB_CHECK(cudaStreamEndCapture(s, &captured));
        BB_CHECK(cudaGraphInstantiate(&made->x, made->g, 0));
        prof_     = saved;
        n_launch_ = n0;
        if (loops_.size() == k_loops)
        {
            loops_.erase(loops_.begin()); // (every tree before this one was waited for)
        }
        loops_.push_back(std::move(made));
        loop = loops_.back().get();
    }
    if (prof_ != nullptr)
    {
        phase_begin();
    }
    BB_CHECK(cudaGraphLaunch(loop->x, s));
    if (prof_ != nullptr)
    {
        phase_end(prof_->other_ms);
    }
    launch_k(pdl_, leaf_loop_end_kernel, 1, k_plan_thr, 0, s, st, cand, leaves_, nodes_[0], ctl_);
    BB_LAUNCH("leaf_loop_end_kernel");
    launches += 1;
    // write_leaf for every leaf, then (quantised) the FP64 renewal, then the
    // rows' leaf ids and score updates from the leaves' segments
    launch_k(pdl_, final_kernel, 1, k_plan_thr, 0, s, ctl_, nodes_[0], tp, t, pchunks_, pcr_,
             nbound_, HeapOut{nullptr, nullptr, 0, 1}, dtree_, tree_step_);
    BB_LAUNCH("final_kernel");
    launches += 1;
    nodes_cur_ = nodes_[0];
    rows_cur_  = rows_[0];
    uint32_t const before = n_launch_;
    leaf_values(t, true);
    launches += n_launch_ - before;
    launch_k(pdl_, stamp_kernel, max_pchunks_, k_threads, 0, s, ctl_, pchunks_, nodes_[0], rows_[0],
             t, leaf_id, scores, lr);
    BB_LAUNCH("stamp_kernel");
    launches += 1;
    // the loop's verdict: a full node table or pool is the reference's
    // capacity refusal
    auto *lh = static_cast<LeafLoop *>(lout_h_);
    BB_CHECK(cudaMemcpyAsync(lh, st, sizeof(LeafLoop), cudaMemcpyDeviceToHost, s));
    BB_CHECK(cudaStreamSynchronize(s));
    if (lh->error == 1)
    {
        throw ConfigError("grower: leafwise tree outgrew its node table");
    }
    if (lh->error == 2)
    {
        throw ConfigError("grower: leafwise histogram pool exhausted");
    }
    if (lh->error == 3)
    {
        throw std::runtime_error("grower: leafwise pop loop exceeded its pop bound");
    }
    // every pop ran the body once (a tree without one ran it empty) -- one
    // graph launch on the host's side
    n_launch_ += launches + std::max(lh->pops, 1u) * body_launches_;
    launches_ = n_launch_;
    ++tree_no_;
}

void Grower::populate(float2 const *gh, uint32_t const *rows, uint32_t n, double2 *out)
{
    cudaStream_t s = stream_;
    gh_cur_        = gh;
    root_rows_     = rows;
    TreeOut t{};
    std::vector<uint32_t> meta_dummy(3);
    // a tree output the setup kernel may write node 0 into
    uint32_t *scratch = dalloc<uint32_t>(64, s);
    t.feature = t.left = t.right = t.split_bin = t.meta = scratch;
    t.value = t.gain = t.cover = reinterpret_cast<float *>(scratch + 16);
    t.default_left = reinterpret_cast<uint8_t *>(scratch + 32);
    if (quant_)
    {
        quantise(gh, static_cast<uint32_t>(plane_.n_rows), false, OpenArgs{});
    }
    walk_   = false;
    chain_  = false;
    packed_ = false;
    launch_k(pdl_, root_setup_kernel, 1, k_threads, 0, s,
             RootArgs{ctl_, nodes_[0], n, bchunks_, brange_, build_, t, crows_, n, nullptr, heap_});
    BB_LAUNCH("root_setup_kernel");
    build(rows, n_sel_, 0, false, 1);
    std::vector<double2> cells(total_cells_);
    if (quant_)
    {
        std::vector<unsigned long long> q(static_cast<size_t>(total_cells_) * cw_);
        double2                         sc{};
        BB_CHECK(cudaMemcpyAsync(q.data(), hist_[0], q.size() * 8ULL, cudaMemcpyDeviceToHost, s));
        BB_CHECK(cudaMemcpyAsync(&sc, qscale_, sizeof(double2), cudaMemcpyDeviceToHost, s));
        BB_CHECK(cudaStreamSynchronize(s));
        for (uint32_t x = 0; x < total_cells_; ++x)
        {
            int64_t const g = cw_ == 2 ? static_cast<int64_t>(q[2 * x])
                                       : static_cast<int32_t>(static_cast<uint32_t>(q[x] >> 32));
            int64_t const h = cw_ == 2 ? static_cast<int64_t>(q[(2 * x) + 1])
                                       : static_cast<int64_t>(static_cast<uint32_t>(q[x]));
            out[x] = make_double2(static_cast<double>(g) * sc.x, static_cast<double>(h) * sc.y);
        }
    }
    else
    {
        std::vector<float2> f(total_cells_);
        BB_CHECK(cudaMemcpyAsync(f.data(), hist_[0], total_cells_ * 8ULL, cudaMemcpyDeviceToHost, s));
        BB_CHECK(cudaStreamSynchronize(s));
        for (uint32_t x = 0; x < total_cells_; ++x)
        {
            out[x] = make_double2(f[x].x, f[x].y);
        }
    }
    BB_CHECK(cudaFreeAsync(scratch, s));
    BB_CHECK(cudaStreamSynchronize(s));
}

void Grower::set_interaction(std::vector<uint64_t> const &fgroups)
{
    if (fgroups_ != nullptr)
    {
        BB_CHECK(cudaFreeAsync(fgroups_, stream_));
        fgroups_ = nullptr;
    }
    if (fgroups.empty())
    {
        return;
    }
    if (cfg_.level)
    {
        // ObliviousGrower refuses them (src/grower_impl.hpp:591-595)
        throw ConfigError("interaction_constraints are not supported by the levelwise grower");
    }
    if (fgroups.size() != plane_.n_feats)
    {
        throw std::invalid_argument("grower: one interaction mask per feature");
    }
    BB_CHECK(cudaMallocAsync(reinterpret_cast<void **>(&fgroups_), fgroups.size() * 8, stream_));
    BB_CHECK(cudaMemcpyAsync(fgroups_, fgroups.data(), fgroups.size() * 8, cudaMemcpyHostToDevice,
                             stream_));
    BB_CHECK(cudaStreamSynchronize(stream_));
}

void Grower::set_monotone(std::vector<int8_t> const &m)
{
    if (mono_ != nullptr)
    {
        BB_CHECK(cudaFreeAsync(mono_, stream_));
        mono_ = nullptr;
    }
    n_mono_ = static_cast<uint32_t>(m.size());
    if (m.empty())
    {
        return;
    }
    BB_CHECK(cudaMallocAsync(reinterpret_cast<void **>(&mono_), m.size(), stream_));
    BB_CHECK(cudaMemcpyAsync(mono_, m.data(), m.size(), cudaMemcpyHostToDevice, stream_));
    BB_CHECK(cudaStreamSynchronize(stream_));
}

} // namespace bb
