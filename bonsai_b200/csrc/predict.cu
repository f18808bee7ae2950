// Ensemble predict: bb_predict_plan_* (pack once, run many) and bb_predict
// (pack, run, release in one call).
//
// The reference packs the ensemble into SoA node tables once
// (cuda_predict_plan, src/cuda/predict.cu:147-196) and walks it with one
// thread per row over every tree, the nodes read from global memory
// (predict_walk_kernel, src/cuda/predict.cu:51-85). Its contract is bit
// equality with the host walk predict_at_binned (include/bonsai/booster.hpp:
// 831-845): each row's leaves summed in float in tree order, then
// init + lr * sum, nothing fused.
//
// Here the ensemble is re-laid for the device as complete binary heaps
// ("heap form"): every tree padded to the ensemble's depth D, a leaf above
// depth D standing in for its whole subtree (its node routes every row left,
// its left descendants repeat it). The root is slot 1 and slot n's children
// are 2n and 2n + 1, so a walk is D unrolled steps with no child tables and
// no exit test, ending on a leaf slot in [2^D, 2^(D+1)). A node is one
// 4-byte word: the byte offset of its feature's code in the row's staged
// codes, and a threshold; the row goes right iff code >= threshold. The
// missing-bin rule of routes_left (include/bonsai/dataset.hpp:234-238)
// becomes the choice of which of two staged variants of the code the node
// reads (the heap node comment below).
//
// Up to depth 8 a lane is a tree and a warp a row (lane_predict_kernel): 32
// trees' heaps lie interleaved, slot by slot, so that a lane's node is in its
// own bank whatever slot it reached, and the row's codes are a few words that
// the lanes share -- one shared-memory wavefront for every load of the walk,
// where a lane per row has conflicts on the lower levels' nodes. A CTA holds a
// tile of rows and streams the trees through shared memory, 32 at a time; the
// 32 values of each row go by shared memory to the row's thread,
// which adds them in tree order. Batches of up to some 1,000 rows take a CTA
// per row, a thread per tree and the nodes straight from L2
// (row_predict_kernel), up to 64 rows several CTAs per row. Depths 9 and 10 take a lane
// per row (heap_predict_kernel), the trees split over CTAs where the rows do not fill
// the GPU, and so do shallow trees over batches that fill its passes. Deeper
// ensembles, or planes wider than 8 mirror tiles (256 u8 / 128 u16 features), use
// the node form: the reference's layout and walk, nodes in global memory.
#include "bonsai_b200.h"
#include "ingest.cuh"

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

struct bb_plane
{
    bb::Plane p;
};

namespace bb
{
namespace
{

constexpr uint32_t k_max_heap_depth = 10;
constexpr uint32_t k_max_heap_tiles = 8;
constexpr uint32_t k_chunk_bytes    = 16384;

void need(bool ok, char const *what)
{
    if (!ok)
    {
        throw std::invalid_argument(what);
    }
}

template <typename F> int guarded(F &&f)
{
    try
    {
        f();
        return BB_OK;
    }
    catch (ConfigError const &e)
    {
        set_last_error(e.what());
        return BB_ERR_CONFIG;
    }
    catch (std::invalid_argument const &e)
    {
        set_last_error(e.what());
        return BB_ERR_ARG;
    }
    catch (std::exception const &e)
    {
        set_last_error(e.what());
        return BB_ERR_CUDA;
    }
}

// ---- heap form ---------------------------------------------------------------

// A heap node: off << 16 | thr. The row's code for the node's feature, in
// the variant its default direction needs, sits at byte off of the row's
// staged codes; the row goes right iff code >= thr. A leaf slot holds the
// leaf value's bits.
//
// Two variants of every code are staged. v1 is the code itself: the missing
// (last) bin is the largest code, so with default_left false "code > split
// or missing" is code >= split + 1. v0 maps the missing bin to 0 and every
// other code c to c + 1: with default_left true "code > split and not
// missing" is v0 >= split + 2. No code reaches the threshold 256 (u8) or
// 65535 (u16), which routes a node left: an always-left pad, or a split that
// sends nothing right.

// The v0 word of a staged v1 word: per code lane, 0 where the code is its
// feature's last bin, else code + 1 (no lane overflows: a non-missing code is
// at most 254, or 65533 for u16).
__device__ __forceinline__ uint32_t missing_low(uint32_t c, uint32_t last, bool u8)
{
    uint32_t const keep = ~(u8 ? __vcmpeq4(c, last) : __vcmpeq2(c, last));
    return (c & keep) + ((u8 ? 0x01010101u : 0x00010001u) & keep);
}

__device__ __forceinline__ uint32_t lds_u32(uint32_t a)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

template <typename CodeT> __device__ __forceinline__ uint32_t lds_code(uint32_t a)
{
    uint32_t v;
    if constexpr (sizeof(CodeT) == 1)
    {
        asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
    }
    else
    {
        asm volatile("ld.shared.u16 %0, [%1];" : "=r"(v) : "r"(a));
    }
    return v;
}

// ---- a lane per tree ----

constexpr uint32_t k_lane_depth   = 8;    // the deepest ensemble taken a lane per tree
constexpr uint32_t k_lane_threads = 512;
constexpr uint32_t k_lane_smem    = 113 * 1024; // two CTAs an SM
constexpr uint32_t k_val_stride   = 33;   // a row's 32 values, rows in different banks
constexpr uint32_t k_row_threads  = 1024;
constexpr uint32_t k_row_vals     = 4096; // values a row's CTA holds at once
constexpr uint32_t k_few_rows     = 64; // up to these, several CTAs per row
constexpr uint32_t k_few_threads  = 128;
constexpr size_t   k_max_smem     = 227 * 1024;
constexpr size_t   k_max_vals     = size_t{256} << 20; // bytes of a split batch's leaf values

__device__ __forceinline__ void cp_async16(void *smem_dst, void const *gsrc)
{
    uint32_t const d = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gsrc));
}

// Word wd of a row's staged codes: v1 words, then v0 words.
__device__ __forceinline__ uint32_t staged_word(uint32_t const *mirror, uint64_t n_rows,
                                                uint64_t row, uint32_t wd, uint32_t words,
                                                uint32_t const *last_words, bool u8)
{
    uint32_t const w1 = wd < words ? wd : wd - words;
    uint32_t const c =
        __ldg(mirror + ((((static_cast<uint64_t>(w1 / 8) * n_rows) + row) * 8) + (w1 % 8)));
    return wd < words ? c : missing_low(c, last_words[w1], u8);
}

// R rows of a warp's tile through its lanes' trees.
template <typename CodeT, uint32_t D, uint32_t R>
__device__ __forceinline__ void lane_walk(unsigned char const *heap, unsigned char const *codes,
                                          uint32_t row_bytes, uint32_t r0, float *vals)
{
    uint32_t const lane4 = (threadIdx.x & 31u) * 4u;
    // byte offsets into the interleaved heaps: slot n of this lane's tree at
    // 128 n + 4 lane, its children at 2p - 4 lane (+ 128)
    uint32_t const cl = 0u - lane4;
    uint32_t const cr = 128u - lane4;
    uint32_t       p[R];
#pragma unroll
    for (uint32_t k = 0; k < R; ++k)
    {
        p[k] = 128u + lane4;
    }
#pragma unroll
    for (uint32_t d = 0; d < D; ++d)
    {
#pragma unroll
        for (uint32_t k = 0; k < R; ++k)
        {
            uint32_t const e = *reinterpret_cast<uint32_t const *>(heap + p[k]);
            uint32_t const c = *reinterpret_cast<CodeT const *>(
                codes + ((r0 + (k_lane_threads / 32 * k)) * row_bytes) + (e >> 16));
            p[k] = (2u * p[k]) + (c >= (e & 0xFFFFu) ? cr : cl);
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < R; ++k)
    {
        vals[((r0 + (k_lane_threads / 32 * k)) * k_val_stride) + (lane4 / 4u)] =
            *reinterpret_cast<float const *>(heap + p[k]);
    }
}

// Scores of rows [blockIdx.x * rows, + rows): warp w takes rows w, w + 16, ...
// through each 32 trees, thread r sums row r. What bounds it is shared-memory
// wavefronts (19 a row and 32 trees at depth 8) and instruction issue, close
// together; two CTAs an SM fill each other's barriers and group loads (one CTA
// of 1,024 threads with two buffers: 3.16 ms for 1,000 trees over 1M rows, two
// so: 2.72; a lane per row, whose lower levels' nodes conflict: 3.21, and 0.78
// against 0.30 at 100,000 rows, where its passes were half empty).
template <typename CodeT, uint32_t D>
__global__ void __launch_bounds__(k_lane_threads, 2)
    lane_predict_kernel(uint32_t const *__restrict__ mirror, uint64_t n_rows, uint32_t n_tiles,
                        uint32_t const *__restrict__ last_words,
                        uint32_t const *__restrict__ heaps, uint32_t n_trees, uint32_t rows,
                        float lr, float init, float *__restrict__ out)
{
    constexpr uint32_t group = 32u * (2u << D) * 4u; // bytes of 32 trees
    constexpr uint32_t warps = k_lane_threads / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned char *const heap_s  = smem;
    float *const         vals_s  = reinterpret_cast<float *>(smem + group);
    uint32_t const       words   = n_tiles * 8;
    unsigned char *const codes_s =
        smem + group + (size_t{rows} * k_val_stride * sizeof(float));
    uint32_t const row_bytes = words * 8;
    uint64_t const row0      = static_cast<uint64_t>(blockIdx.x) * rows;
    uint32_t const live      = static_cast<uint32_t>(min(static_cast<uint64_t>(rows), n_rows - row0));
    uint32_t const warp      = threadIdx.x >> 5;
    uint32_t const groups    = (n_trees + 31) / 32;
    auto const     load      = [&](uint32_t c)
    {
        auto const *src = reinterpret_cast<unsigned char const *>(heaps) +
                          (static_cast<size_t>(c) * group);
        for (uint32_t i = threadIdx.x * 16u; i < group; i += k_lane_threads * 16u)
        {
            cp_async16(heap_s + i, src + i);
        }
    };
    load(0);
    for (uint32_t i = threadIdx.x; i < live * 2 * words; i += k_lane_threads)
    {
        uint32_t const r = i / (2 * words);
        reinterpret_cast<uint32_t *>(codes_s)[i] = staged_word(
            mirror, n_rows, row0 + r, i - (r * 2 * words), words, last_words, sizeof(CodeT) == 1);
    }
    float acc = 0.0F;
    for (uint32_t c = 0; c < groups; ++c)
    {
        asm volatile("cp.async.wait_all;\n" ::);
        __syncthreads(); // the group is here (and the codes; the last values are added)
        for (uint32_t r0 = warp; r0 < live; r0 += 4 * warps)
        {
            // (the same for the whole warp)
            uint32_t const left = (live - r0 + warps - 1) / warps;
            if (left >= 4)
            {
                lane_walk<CodeT, D, 4>(heap_s, codes_s, row_bytes, r0, vals_s);
            }
            else if (left == 3)
            {
                lane_walk<CodeT, D, 3>(heap_s, codes_s, row_bytes, r0, vals_s);
            }
            else if (left == 2)
            {
                lane_walk<CodeT, D, 2>(heap_s, codes_s, row_bytes, r0, vals_s);
            }
            else
            {
                lane_walk<CodeT, D, 1>(heap_s, codes_s, row_bytes, r0, vals_s);
            }
        }
        __syncthreads(); // the values are here, the group is done with
        if (c + 1 < groups)
        {
            load(c + 1);
        }
        if (threadIdx.x < live)
        {
            float const   *v = vals_s + (threadIdx.x * k_val_stride);
            uint32_t const m = min(32u, n_trees - (c * 32));
            if (m == 32)
            {
#pragma unroll
                for (uint32_t t = 0; t < 32; ++t)
                {
                    acc = acc + v[t];
                }
            }
            else
            {
                for (uint32_t t = 0; t < m; ++t)
                {
                    acc = acc + v[t];
                }
            }
        }
    }
    if (threadIdx.x < live)
    {
        out[row0 + threadIdx.x] = __fadd_rn(init, __fmul_rn(acc, lr));
    }
}

// A thread's tree for a row whose staged codes are in shared memory, nodes
// from global memory (a warp's 32 trees side by side): the leaf's value.
template <typename CodeT>
__device__ __forceinline__ float tree_value(uint32_t const *__restrict__ heaps, uint32_t t,
                                            uint32_t D, uint32_t const *codes_s)
{
    uint32_t const *h = heaps + ((t / 32) * (size_t{32} * (2u << D))) + (t % 32);
    uint32_t        n = 1;
    for (uint32_t d = 0; d < D; ++d)
    {
        uint32_t const e = __ldg(h + (n * 32));
        uint32_t const c = *reinterpret_cast<CodeT const *>(
            reinterpret_cast<unsigned char const *>(codes_s) + (e >> 16));
        n = (2 * n) + (c >= (e & 0xFFFFu) ? 1 : 0);
    }
    return __uint_as_float(__ldg(h + (n * 32)));
}

// m values of shared memory (16-byte aligned) onto acc, in order.
__device__ __forceinline__ float add_values(float acc, float const *vals_s, uint32_t m)
{
    uint32_t i = 0;
#pragma unroll 4
    for (; i + 4 <= m; i += 4)
    {
        float4 const v = *reinterpret_cast<float4 const *>(vals_s + i);
        acc            = acc + v.x;
        acc            = acc + v.y;
        acc            = acc + v.z;
        acc            = acc + v.w;
    }
    for (; i < m; ++i)
    {
        acc = acc + vals_s[i];
    }
    return acc;
}

template <typename CodeT>
__device__ __forceinline__ void stage_row(uint32_t *codes_s, uint32_t const *mirror,
                                          uint64_t n_rows, uint64_t row, uint32_t n_tiles,
                                          uint32_t const *last_words)
{
    uint32_t const words = n_tiles * 8;
    for (uint32_t i = threadIdx.x; i < 2 * words; i += blockDim.x)
    {
        codes_s[i] =
            staged_word(mirror, n_rows, row, i, words, last_words, sizeof(CodeT) == 1);
    }
    __syncthreads();
}

// A CTA per row, a thread per tree; then one thread adds the values in tree
// order.
template <typename CodeT>
__global__ void __launch_bounds__(k_row_threads)
    row_predict_kernel(uint32_t const *__restrict__ mirror, uint64_t n_rows, uint32_t n_tiles,
                       uint32_t const *__restrict__ last_words,
                       uint32_t const *__restrict__ heaps, uint32_t D, uint32_t n_trees, float lr,
                       float init, float *__restrict__ out)
{
    __shared__ __align__(16) float    vals_s[k_row_vals];
    __shared__ __align__(16) uint32_t codes_s[k_max_heap_tiles * 16];
    stage_row<CodeT>(codes_s, mirror, n_rows, blockIdx.x, n_tiles, last_words);
    float acc = 0.0F;
    for (uint32_t t0 = 0; t0 < n_trees; t0 += k_row_vals)
    {
        uint32_t const m = min(k_row_vals, n_trees - t0);
        for (uint32_t i = threadIdx.x; i < m; i += blockDim.x)
        {
            vals_s[i] = tree_value<CodeT>(heaps, t0 + i, D, codes_s);
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            acc = add_values(acc, vals_s, m);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        out[blockIdx.x] = __fadd_rn(init, __fmul_rn(acc, lr));
    }
}

// The fewest rows: the trees of a row over several CTAs (one SM's load path
// bounds a row's 1,000 walks), every value kept, then a CTA per row sums them
// in tree order.
template <typename CodeT>
__global__ void __launch_bounds__(k_few_threads)
    few_values_kernel(uint32_t const *__restrict__ mirror, uint64_t n_rows, uint32_t n_tiles,
                      uint32_t const *__restrict__ last_words,
                      uint32_t const *__restrict__ heaps, uint32_t D, uint32_t n_trees,
                      float *__restrict__ vals)
{
    __shared__ __align__(16) uint32_t codes_s[k_max_heap_tiles * 16];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); // the sum may be set up
    stage_row<CodeT>(codes_s, mirror, n_rows, blockIdx.x, n_tiles, last_words);
    uint32_t const t = (blockIdx.y * k_few_threads) + threadIdx.x;
    if (t < n_trees)
    {
        vals[(static_cast<uint64_t>(blockIdx.x) * n_trees) + t] =
            tree_value<CodeT>(heaps, t, D, codes_s);
    }
}

__global__ void __launch_bounds__(k_few_threads)
    few_sum_kernel(float const *vals, uint32_t n_trees, float lr, float init,
                   float *__restrict__ out)
{
    __shared__ __align__(16) float vals_s[k_row_vals];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float const *row = vals + (static_cast<uint64_t>(blockIdx.x) * n_trees);
    float        acc = 0.0F;
    for (uint32_t t0 = 0; t0 < n_trees; t0 += k_row_vals)
    {
        uint32_t const m = min(k_row_vals, n_trees - t0);
        for (uint32_t i = threadIdx.x; i < m; i += k_few_threads)
        {
            vals_s[i] = __ldcg(row + t0 + i);
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            acc = add_values(acc, vals_s, m);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0)
    {
        out[blockIdx.x] = __fadd_rn(init, __fmul_rn(acc, lr));
    }
}

// ---- a lane per row (depths 9 and 10, and full waves of shallow trees) ----

// BY32: the heaps are those of the lane-per-tree form (32 trees interleaved, a
// row's words one after another) and are turned while they are staged: each
// tree's slots together, an odd stride from tree to tree, the code offsets
// for a lane's column of the staged codes.
// Scores of rows [blockIdx.x * rows_per_cta, + rows_per_cta), taken T x R
// rows at a time: out[r] = init + lr * sum. SPLIT, with vals not null: the trees
// [blockIdx.y * trees_per_split, + trees_per_split) only, every (tree, row) leaf
// value into vals[t * n_rows + r].
template <typename CodeT, uint32_t D, uint32_t T, uint32_t R, bool BY32, bool SPLIT>
__global__ void __launch_bounds__(T)
    heap_predict_kernel(uint4 const *__restrict__ mirror, uint64_t n_rows, uint32_t n_tiles,
                        uint32_t const *__restrict__ last_words,
                        uint32_t const *__restrict__ heaps, uint32_t n_trees,
                        uint32_t chunk_trees, uint32_t rows_per_cta, float lr, float init,
                        float *__restrict__ out, uint32_t trees_per_split,
                        float *__restrict__ vals)
{
    constexpr uint32_t slots = 2u << D; // per tree: root at 1, leaves at [2^D, 2^(D+1))
    constexpr uint32_t pitch = slots + (BY32 ? 1u : 0u);
    constexpr uint32_t warps = T / 32;
    constexpr bool     u8    = sizeof(CodeT) == 1;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t const words  = n_tiles * 8;     // v1 words per row; v0 follows
    uint32_t const lane   = threadIdx.x & 31u;
    uint32_t const warp   = threadIdx.x >> 5;
    auto *const    codes  = smem;
    auto *const    heap_s = reinterpret_cast<uint32_t *>(
        smem + (static_cast<size_t>(T) * R * words * 8));
    uint32_t const codes_a =
        static_cast<uint32_t>(__cvta_generic_to_shared(codes));
    uint32_t const heap_a = static_cast<uint32_t>(__cvta_generic_to_shared(heap_s));
    uint64_t const begin = static_cast<uint64_t>(blockIdx.x) * rows_per_cta;
    uint64_t const end   = min(n_rows, begin + rows_per_cta);
    uint32_t const t0    = SPLIT ? blockIdx.y * trees_per_split : 0;
    uint32_t const t1    = SPLIT ? min(n_trees, t0 + trees_per_split) : n_trees;

    for (uint64_t row0 = begin; row0 < end; row0 += T * R)
    {
        // this thread's rows: slot s = warp + 8k holds 32 consecutive rows;
        // word j of a row in lane l sits at word (s * 2 words + j) * 32 + l
        uint64_t row[R];
        uint32_t base[R];
        __syncthreads(); // the previous pass's walks are done with the codes
#pragma unroll
        for (uint32_t k = 0; k < R; ++k)
        {
            uint32_t const s = warp + (warps * k);
            row[k]           = row0 + (s * 32u) + lane;
            base[k]          = codes_a + (((s * words * 64u) + lane) * 4u);
            auto *cw = reinterpret_cast<uint32_t *>(codes) + (s * words * 64u) + lane;
            for (uint32_t t = 0; t < n_tiles; ++t)
            {
                uint4 x = make_uint4(0, 0, 0, 0);
                uint4 y = make_uint4(0, 0, 0, 0);
                if (row[k] < end)
                {
                    uint4 const *src =
                        mirror + (((static_cast<uint64_t>(t) * n_rows) + row[k]) * 2);
                    x = src[0];
                    y = src[1];
                }
                uint32_t const w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j)
                {
                    uint32_t const wd = (t * 8u) + j;
                    cw[wd * 32u]           = w[j];
                    cw[(words + wd) * 32u] = missing_low(w[j], last_words[wd], u8);
                }
            }
        }
        float acc[R];
#pragma unroll
        for (uint32_t k = 0; k < R; ++k)
        {
            acc[k] = 0.0F;
        }
        for (uint32_t c0 = t0; c0 < t1; c0 += chunk_trees)
        {
            uint32_t const nc = min(chunk_trees, t1 - c0);
            __syncthreads(); // codes staged; the previous chunk's walks done
            if constexpr (BY32)
            {
                // four trees' words of a slot at a time; a chunk is whole
                // groups of 32 trees, or a part of one
                auto const *src  = reinterpret_cast<uint4 const *>(heaps);
                auto const  turn = [](uint32_t e, bool inner)
                { return inner ? ((e & 0xFFFC0000u) << 5) | (e & 0x3FFFFu) : e; };
                uint32_t const wide = min(8u, chunk_trees / 4u);
                uint32_t const q0   = c0 / 4u;
                uint32_t const n16  = ((nc + (4u * wide) - 1) / (4u * wide)) * slots * wide;
                for (uint32_t i = threadIdx.x; i < n16; i += T)
                {
                    uint32_t const sub   = i % wide;
                    uint32_t const slot  = (i / wide) % slots;
                    uint32_t const blk   = i / (wide * slots);
                    uint4 const    x     = src[(((((q0 / 8u) + blk) * slots) + slot) * 8u) +
                                        (q0 % 8u) + sub];
                    bool const     inner = slot < (1u << D);
                    uint32_t      *dst   = heap_s + (((blk * 32u) + (sub * 4u)) * pitch) + slot;
                    dst[0]               = turn(x.x, inner);
                    dst[pitch]           = turn(x.y, inner);
                    dst[2 * pitch]       = turn(x.z, inner);
                    dst[3 * pitch]       = turn(x.w, inner);
                }
            }
            else
            {
                auto const *src =
                    reinterpret_cast<uint4 const *>(heaps + (static_cast<size_t>(c0) * slots));
                auto          *dst = reinterpret_cast<uint4 *>(heap_s);
                uint32_t const n16 = nc * slots / 4u;
                for (uint32_t i = threadIdx.x; i < n16; i += T)
                {
                    dst[i] = src[i];
                }
            }
            __syncthreads();
            for (uint32_t j = 0; j < nc; ++j)
            {
                // byte addresses in the shared window: slot i of this tree
                // at tb + 4i; from p = tb + 4n the child 2n (+1) is
                // 2p - tb (+4)
                uint32_t const tb = heap_a + (j * pitch * 4u);
                uint32_t const cl = 0u - tb;
                uint32_t const cr = 4u - tb;
                uint32_t p[R];
#pragma unroll
                for (uint32_t k = 0; k < R; ++k)
                {
                    p[k] = tb + 4u;
                }
#pragma unroll
                for (uint32_t d = 0; d < D; ++d)
                {
#pragma unroll
                    for (uint32_t k = 0; k < R; ++k)
                    {
                        uint32_t const e    = lds_u32(p[k]);
                        uint32_t const code = lds_code<CodeT>(base[k] + (e >> 16));
                        p[k] = (2u * p[k]) + (code >= (e & 0xFFFFu) ? cr : cl);
                    }
                }
#pragma unroll
                for (uint32_t k = 0; k < R; ++k)
                {
                    float const v = __uint_as_float(lds_u32(p[k]));
                    if (!SPLIT || vals == nullptr)
                    {
                        acc[k] = acc[k] + v;
                    }
                    else if (row[k] < end)
                    {
                        vals[(static_cast<uint64_t>(c0 + j) * n_rows) + row[k]] = v;
                    }
                }
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < R; ++k)
        {
            if (row[k] < end && (!SPLIT || vals == nullptr))
            {
                out[row[k]] = __fadd_rn(init, __fmul_rn(acc[k], lr));
            }
        }
    }
}

// Every row's leaf values summed in tree order: one thread per row.
__global__ void sum_rows_kernel(float const *__restrict__ vals, uint64_t n_rows, uint32_t n_trees,
                                float lr, float init, float *__restrict__ out)
{
    uint64_t const r = (static_cast<uint64_t>(blockIdx.x) * blockDim.x) + threadIdx.x;
    if (r >= n_rows)
    {
        return;
    }
    float acc = 0.0F;
#pragma unroll 8
    for (uint32_t t = 0; t < n_trees; ++t)
    {
        acc = acc + vals[(static_cast<uint64_t>(t) * n_rows) + r];
    }
    out[r] = __fadd_rn(init, __fmul_rn(acc, lr));
}

// The same sum with one warp per row, for batches too small to fill the GPU
// with rows: lanes load 32 trees' values at once, every lane adds them in
// order from the shuffles.
__global__ void sum_warp_kernel(float const *__restrict__ vals, uint64_t n_rows, uint32_t n_trees,
                                float lr, float init, float *__restrict__ out)
{
    uint64_t const r    = ((static_cast<uint64_t>(blockIdx.x) * blockDim.x) + threadIdx.x) >> 5;
    uint32_t const lane = threadIdx.x & 31u;
    if (r >= n_rows)
    {
        return;
    }
    float acc = 0.0F;
    for (uint32_t t0 = 0; t0 < n_trees; t0 += 32)
    {
        uint32_t const m = min(32u, n_trees - t0);
        float const    v = lane < m ? vals[(static_cast<uint64_t>(t0 + lane) * n_rows) + r] : 0.0F;
        for (uint32_t j = 0; j < m; ++j)
        {
            acc = acc + __shfl_sync(0xFFFFFFFFu, v, static_cast<int>(j));
        }
    }
    if (lane == 0)
    {
        out[r] = __fadd_rn(init, __fmul_rn(acc, lr));
    }
}

// ---- node form (deep trees, wide planes) ---------------------------------------

// One thread per row, every tree in order: the bin-space walk of
// routes_left over tree-local child ids, nodes in global memory.
template <typename BinT>
__global__ void node_predict_kernel(BinT const *__restrict__ bins, uint64_t n_pad, uint64_t n,
                                    uint32_t const *__restrict__ last_bin, uint32_t n_trees,
                                    uint32_t const *__restrict__ roots,
                                    uint32_t const *__restrict__ feature,
                                    uint32_t const *__restrict__ split_bin,
                                    uint32_t const *__restrict__ left,
                                    uint32_t const *__restrict__ right,
                                    uint8_t const *__restrict__ dl,
                                    float const *__restrict__ value, float lr, float init,
                                    float *__restrict__ out)
{
    uint64_t const r = (static_cast<uint64_t>(blockIdx.x) * blockDim.x) + threadIdx.x;
    if (r >= n)
    {
        return;
    }
    float acc = 0.0F;
    for (uint32_t t = 0; t < n_trees; ++t)
    {
        uint32_t const base = roots[t];
        uint32_t       idx  = base;
        while (feature[idx] != k_leaf_flag)
        {
            uint32_t const f = feature[idx];
            uint32_t const b = bins[(static_cast<uint64_t>(f) * n_pad) + r];
            idx = base + (routes_left(b, last_bin[f], split_bin[idx], dl[idx] != 0) ? left[idx]
                                                                                   : right[idx]);
        }
        acc = acc + value[idx];
    }
    out[r] = __fadd_rn(init, __fmul_rn(acc, lr));
}

// ---- host packing ---------------------------------------------------------------

} // namespace

// A device buffer released with its owner.
struct DeviceBuf
{
    void  *p   = nullptr;
    size_t cap = 0;
    DeviceBuf() = default;
    DeviceBuf(DeviceBuf const &) = delete;
    DeviceBuf &operator=(DeviceBuf const &) = delete;
    ~DeviceBuf()
    {
        if (p != nullptr)
        {
            cudaFree(p);
        }
    }
    void alloc(size_t bytes)
    {
        check(cudaMalloc(&p, std::max<size_t>(bytes, 16)), "cudaMalloc");
        cap = std::max<size_t>(bytes, 16);
    }
    // At least this many bytes, whatever they hold.
    void grow(size_t bytes)
    {
        if (cap < bytes)
        {
            if (p != nullptr)
            {
                check(cudaFree(p), "cudaFree");
                p   = nullptr;
                cap = 0;
            }
            alloc(bytes);
        }
    }
    void upload(void const *src, size_t bytes)
    {
        alloc(bytes);
        check(cudaMemcpy(p, src, bytes, cudaMemcpyHostToDevice), "cudaMemcpy");
    }
    template <typename T> T *as() const
    {
        return static_cast<T *>(p);
    }
};

} // namespace bb

struct bb_predict_plan
{
    // the plane shape the ensemble was packed for
    uint32_t              n_feats = 0;
    bool                  u8      = true;
    std::vector<uint32_t> cut_off;
    uint32_t              n_trees = 0;
    float                 lr      = 0.0F;
    float                 init    = 0.0F;
    // heap form (depth > 0) or node form (depth == 0)
    uint32_t    depth   = 0;
    uint32_t    n_tiles = 0;
    uint32_t    sms     = 1;
    uint32_t    lane_rows = 0; // a lane CTA's most rows
    uint64_t    heap_ctas = 0; // resident CTAs of the lane-per-row form; 0: not taken
    bb::DeviceBuf tables; // of the heap form, in one allocation:
    uint32_t     *heaps      = nullptr;
    uint32_t     *last_words = nullptr; // per staged code word, its features' last bins
    float        *few_vals   = nullptr; // a few rows' leaf values (depths to 8)
    bb::DeviceBuf vals;                 // a split batch's leaf values (depths 9, 10)
    bb::DeviceBuf last, roots, feature, split, left, right, dl, value;
    // the host runs' output, grown on demand; runs through one plan serialise
    std::mutex   mu;
    float       *out      = nullptr;
    size_t       out_cap  = 0;
    cudaStream_t stream   = nullptr;
    ~bb_predict_plan()
    {
        if (out != nullptr)
        {
            cudaFree(out);
        }
        if (stream != nullptr)
        {
            cudaStreamDestroy(stream);
        }
    }
};

namespace bb
{
namespace
{

void validate_trees(Plane const &p, uint32_t n_trees, uint32_t const *roots, uint32_t n_nodes,
                    uint32_t const *feature, uint32_t const *left, uint32_t const *right)
{
    // every walk must end: children lie after their parent inside the tree,
    // and split features exist
    for (uint32_t t = 0; t < n_trees; ++t)
    {
        uint32_t const b = roots[t];
        uint32_t const e = t + 1 < n_trees ? roots[t + 1] : n_nodes;
        need(b < e && e <= n_nodes, "bb_predict: bad tree roots");
        for (uint32_t i = b; i < e; ++i)
        {
            if (feature[i] == k_leaf_flag)
            {
                continue;
            }
            need(feature[i] < p.n_feats, "bb_predict: node feature out of range");
            need(left[i] > i - b && right[i] > i - b && b + left[i] < e && b + right[i] < e,
                 "bb_predict: a child id must follow its parent in its tree");
        }
    }
}

// Longest root-to-leaf path of tree [b, e) (children follow parents, so one
// pass in id order settles every node's depth).
uint32_t tree_depth(uint32_t b, uint32_t e, uint32_t const *feature, uint32_t const *left,
                    uint32_t const *right)
{
    std::vector<uint32_t> d(e - b, 0);
    uint32_t              deepest = 0;
    for (uint32_t i = 0; i < e - b; ++i)
    {
        deepest = std::max(deepest, d[i]);
        if (feature[b + i] != k_leaf_flag)
        {
            d[left[b + i]]  = std::max(d[left[b + i]], d[i] + 1);
            d[right[b + i]] = std::max(d[right[b + i]], d[i] + 1);
        }
    }
    return deepest;
}

// One tree into its heap: node thresholds and code offsets for a plane of
// u8 (or u16) codes with `words` staged v1 words per row.
struct HeapPacker
{
    uint32_t        D;
    bool            u8;
    uint32_t        words;
    bool            lanes;  // a lane per tree: the row's words one after another
    uint32_t        stride; // words from a heap slot to the next
    uint32_t const *cut_off;
    uint32_t const *feature;
    uint32_t const *split;
    uint32_t const *left;
    uint32_t const *right;
    uint8_t const  *dl;
    float const    *value;

    uint32_t never() const
    {
        return u8 ? 256u : 65535u;
    }
    // Byte offset of feature f's code in the staged row, variant v1 or v0.
    uint32_t code_offset(uint32_t f, bool v0) const
    {
        uint32_t const wd = u8 ? f >> 2 : f >> 1;
        uint32_t const b  = u8 ? f & 3u : (f & 1u) * 2u;
        return (((v0 ? words : 0u) + wd) * (lanes ? 4u : 128u)) + b;
    }
    // routes_left(code, last, split, dl) == !(variant code >= thr).
    uint32_t route(uint32_t f, uint32_t split_bin, bool default_left, uint32_t last) const
    {
        if (split_bin >= last)
        {
            // only the missing bin can go right, and only with default_left false
            return default_left ? never() : (code_offset(f, false) << 16) | last;
        }
        if (default_left)
        {
            return (code_offset(f, true) << 16) | (split_bin + 2);
        }
        return (code_offset(f, false) << 16) | (split_bin + 1);
    }
    static uint32_t leaf_slot(float v)
    {
        uint32_t u = 0;
        std::memcpy(&u, &v, 4);
        return u;
    }
    // Node i (global id; b its tree's first) into heap slot h at depth d (slot h lies
    // at heap[h * stride])
    void fill(uint32_t *heap, uint32_t b, uint32_t i, uint32_t h, uint32_t d) const
    {
        if (d == D)
        {
            heap[size_t{h} * stride] = leaf_slot(value[i]);
            return;
        }
        if (feature[i] == k_leaf_flag)
        {
            // a leaf above depth D: route everything left, repeat it below
            heap[size_t{h} * stride] = never();
            fill(heap, b, i, 2 * h, d + 1);
            fill(heap, b, i, (2 * h) + 1, d + 1);
            return;
        }
        uint32_t const f = feature[i];
        heap[size_t{h} * stride] = route(f, split[i], dl[i] != 0, cut_off[f + 1] - cut_off[f] - 1);
        fill(heap, b, b + left[i], 2 * h, d + 1);
        fill(heap, b, b + right[i], (2 * h) + 1, d + 1);
    }
};

void plan_check_plane(bb_predict_plan const &pl, Plane const &p)
{
    need(p.n_feats == pl.n_feats && p.u8 == pl.u8,
         "bb_predict_plan: the plane's shape differs from the plan's");
    need(std::equal(pl.cut_off.begin(), pl.cut_off.end(), p.h_cut_off),
         "bb_predict_plan: the plane's bin counts differ from the plan's");
}

using HeapFn = void (*)(uint4 const *, uint64_t, uint32_t, uint32_t const *, uint32_t const *,
                        uint32_t, uint32_t, uint32_t, float, float, float *, uint32_t, float *);

// The shapes of a lane per row: 512 threads of two rows, and for depths 9 and 10
// 256 of one, whose codes leave room on planes of four to eight mirror tiles.
template <typename CodeT> HeapFn heap_fn_d(uint32_t D, uint32_t T)
{
    if (T == 256)
    {
        return D == 9 ? heap_predict_kernel<CodeT, 9, 256, 1, false, true>
                      : heap_predict_kernel<CodeT, 10, 256, 1, false, true>;
    }
    switch (D)
    {
    case 1: return heap_predict_kernel<CodeT, 1, 512, 2, true, false>;
    case 2: return heap_predict_kernel<CodeT, 2, 512, 2, true, false>;
    case 3: return heap_predict_kernel<CodeT, 3, 512, 2, true, false>;
    case 4: return heap_predict_kernel<CodeT, 4, 512, 2, true, false>;
    case 5: return heap_predict_kernel<CodeT, 5, 512, 2, true, false>;
    case 6: return heap_predict_kernel<CodeT, 6, 512, 2, true, false>;
    case 7: return heap_predict_kernel<CodeT, 7, 512, 2, true, false>;
    case 8: return heap_predict_kernel<CodeT, 8, 512, 2, true, false>;
    case 9: return heap_predict_kernel<CodeT, 9, 512, 2, false, false>;
    case 10: return heap_predict_kernel<CodeT, 10, 512, 2, false, false>;
    default: throw std::logic_error("bb_predict_plan: heap depth out of range");
    }
}

HeapFn heap_fn(bool u8, uint32_t D, uint32_t T)
{
    return u8 ? heap_fn_d<uint8_t>(D, T) : heap_fn_d<uint16_t>(D, T);
}

// A lane per row: the trees of a chunk, and the shared memory of a CTA of T
// threads (both code variants, 64 bytes a row and mirror tile) with it.
uint32_t heap_chunk(uint32_t D)
{
    uint32_t const tree_bytes = (2u << D) * 4u;
    uint32_t const chunk      = std::max(1u, k_chunk_bytes / tree_bytes);
    // (depth 8: half a group of 32, depth 7: one; of 16 KB, 8 and 16 trees, whose
    // reads are not whole lines, a pass took 8% and 4% longer)
    return D <= 6 ? chunk & ~31u : (D <= k_lane_depth ? 2 * chunk : chunk);
}

size_t heap_smem(uint32_t D, uint32_t n_tiles, uint32_t T)
{
    size_t const tree_bytes = ((2u << D) + (D <= k_lane_depth ? 1u : 0u)) * 4u;
    return (size_t{T == 512 ? 1024u : T} * n_tiles * 64) + (heap_chunk(D) * tree_bytes);
}

// The larger shape whose rows' codes fit.
uint32_t heap_threads(uint32_t D, uint32_t n_tiles)
{
    return heap_smem(D, n_tiles, 512) <= k_max_smem ? 512 : 256;
}

using LaneFn = void (*)(uint32_t const *, uint64_t, uint32_t, uint32_t const *, uint32_t const *,
                        uint32_t, uint32_t, float, float, float *);

template <typename CodeT> LaneFn lane_fn_d(uint32_t D)
{
    switch (D)
    {
    case 1: return lane_predict_kernel<CodeT, 1>;
    case 2: return lane_predict_kernel<CodeT, 2>;
    case 3: return lane_predict_kernel<CodeT, 3>;
    case 4: return lane_predict_kernel<CodeT, 4>;
    case 5: return lane_predict_kernel<CodeT, 5>;
    case 6: return lane_predict_kernel<CodeT, 6>;
    case 7: return lane_predict_kernel<CodeT, 7>;
    case 8: return lane_predict_kernel<CodeT, 8>;
    default: throw std::logic_error("bb_predict_plan: lane depth out of range");
    }
}

LaneFn lane_fn(bool u8, uint32_t D)
{
    return u8 ? lane_fn_d<uint8_t>(D) : lane_fn_d<uint16_t>(D);
}

// Shared memory of a lane CTA over `rows` rows.
size_t lane_smem(uint32_t D, uint32_t n_tiles, uint32_t rows)
{
    return (size_t{32} * (2u << D) * 4) +
           (size_t{rows} * ((k_val_stride * sizeof(float)) + (n_tiles * 64)));
}

uint32_t sm_count()
{
    int dev = 0;
    int n   = 0;
    check(cudaGetDevice(&dev), "cudaGetDevice");
    check(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
    return static_cast<uint32_t>(std::max(n, 1));
}

// Whether a batch takes a CTA per row: while the rows' CTAs of 256 threads all
// run at once, eight an SM, and over two such waves where there are many trees,
// which every CTA of the lane-per-tree form streams whole. (28 features, device
// us a CTA per row / a lane per tree: 1,000 trees of depth 8, 1,100 rows 22.8 / 41.3,
// 1,700 rows 39.4 / 42.0, 2,500 rows 55.2 / 43.3; 300 trees of depth 8, 1,100 rows
// 11.7 / 16.7, 1,700 rows 18.8 / 16.8.)
bool row_form(uint64_t n, uint32_t n_trees, uint32_t sms)
{
    uint64_t const wave = uint64_t{8} * sms;
    return n <= wave || (n <= 2 * wave && n_trees > 500);
}

// Threads of a row's CTA: the most, up to 1,024, that let every row's CTA run at
// once. (1,000 trees of depth 8 over 1,000 rows: 38.8 us with 1,024, 28.9 with 512,
// 20.9 with 256; over 150 rows 12.5, 12.6, 14.6.)
uint32_t row_threads(uint64_t n, uint32_t sms)
{
    uint32_t T = k_row_threads;
    while (T > 256 && n * T > uint64_t{2048} * sms)
    {
        T /= 2;
    }
    return T;
}

// A lane per row: one wave of resident CTAs, each over an equal run of rows.
uint32_t heap_launch(bb_predict_plan &pl, Plane const &p, uint32_t n_trees, float *out,
                     cudaStream_t s)
{
    uint64_t const n   = p.n_rows;
    uint32_t const T   = heap_threads(pl.depth, pl.n_tiles);
    uint64_t const per = std::max<uint64_t>(
        32, ((((n + pl.heap_ctas - 1) / pl.heap_ctas) + 31) / 32) * 32);
    heap_fn(pl.u8, pl.depth, T)<<<ceil_div(n, per), T, heap_smem(pl.depth, pl.n_tiles, T), s>>>(
        static_cast<uint4 const *>(p.mirror), n, pl.n_tiles, pl.last_words,
        pl.heaps, n_trees, heap_chunk(pl.depth), static_cast<uint32_t>(per), pl.lr,
        pl.init, out, n_trees, nullptr);
    BB_LAUNCH("heap_predict_kernel");
    return 1;
}

// Depths 9 and 10 where the rows alone leave SMs idle: the trees split over CTAs
// of 256 rows, every leaf value kept, then summed in tree order. (500 trees of
// depth 10 over 28 features, 64 / 4,000 / 30,000 rows: 31 / 60 / 192 us; a wave
// of CTAs that each take every tree 379 / 383 / 585.)
uint32_t split_launch(bb_predict_plan &pl, Plane const &p, uint32_t n_trees, float *out,
                      cudaStream_t s)
{
    uint64_t const n        = p.n_rows;
    uint32_t const chunk    = heap_chunk(pl.depth);
    uint32_t const row_blks = ceil_div(n, 256);
    uint32_t const n_chunks = ceil_div(n_trees, chunk);
    uint32_t       splits   = std::min(ceil_div(2 * pl.sms, row_blks), n_chunks);
    uint32_t const tps      = ceil_div(ceil_div(n_trees, splits), chunk) * chunk;
    splits                  = ceil_div(n_trees, tps);
    float *vals             = nullptr;
    if (splits > 1)
    {
        pl.vals.grow(n * static_cast<size_t>(n_trees) * sizeof(float));
        vals = pl.vals.as<float>();
    }
    heap_fn(pl.u8, pl.depth, 256)<<<dim3(row_blks, splits), 256,
                                    heap_smem(pl.depth, pl.n_tiles, 256), s>>>(
        static_cast<uint4 const *>(p.mirror), n, pl.n_tiles, pl.last_words,
        pl.heaps, n_trees, chunk, 256, pl.lr, pl.init, out, tps, vals);
    BB_LAUNCH("heap_predict_kernel");
    if (splits == 1)
    {
        return 1;
    }
    if (n < 4096)
    {
        sum_warp_kernel<<<ceil_div(n * 32, 256), 256, 0, s>>>(vals, n, n_trees, pl.lr, pl.init,
                                                              out);
    }
    else
    {
        sum_rows_kernel<<<ceil_div(n, 256), 256, 0, s>>>(vals, n, n_trees, pl.lr, pl.init, out);
    }
    BB_LAUNCH("predict sum kernel");
    return 2;
}

// Whether a lane per row is the faster form at depths up to k_lane_depth. It has
// no step between a walk's end and the sum, but takes whole passes of 1,024
// rows a CTA. Measured at full passes, picoseconds a row over all SMs: about
// 34 + 0.31 x trees x depth (0.33 at depth 8, staged in half lines), and a fifth
// more with two mirror tiles; a lane per tree: 20 and, for every 32 trees,
// 25 + 7 x depth. (589,039 rows, 100 trees of depth 4 / 250 of depth 5: 84 / 236 us
// a lane per row, 132 / 279 a lane per tree; 150,000 rows, half a pass: 55 / 132
// and 44 / 86; 300,000 rows, 1,000 trees of depth 8: 885 and 811.)
bool by_row(bb_predict_plan const &pl, uint64_t n, uint32_t n_trees)
{
    uint64_t const pass   = uint64_t{1024} * pl.heap_ctas;
    double const   passes = static_cast<double>(((n + pass - 1) / pass) * pass);
    double const   node   = pl.depth == 8 ? 0.333 : 0.31;
    double const   row =
        passes * (34.0 + (node * n_trees * pl.depth)) * (pl.n_tiles > 1 ? 1.2 : 1.0);
    double const   tree =
        static_cast<double>(n) * (20.0 + (25.0 * (pl.n_tiles - 1)) +
                                  (((n_trees + 31) / 32) * (25.0 + (7.0 * pl.depth))));
    return row < tree;
}

// Enqueues the scores of the plan's first n_trees trees over plane p into
// out (device, n_rows floats) on stream s. Returns the kernel launches made.
uint32_t plan_launch(bb_predict_plan &pl, Plane const &p, uint32_t n_trees, float *out,
                     cudaStream_t s)
{
    uint64_t const n = p.n_rows;
    if (n == 0)
    {
        return 0; // an empty request plane: nothing to score
    }
    if (pl.depth == 0)
    {
        if (p.u8)
        {
            node_predict_kernel<uint8_t><<<ceil_div(n, 256), 256, 0, s>>>(
                static_cast<uint8_t const *>(p.bins), p.n_pad, n, pl.last.as<uint32_t>(),
                n_trees, pl.roots.as<uint32_t>(), pl.feature.as<uint32_t>(),
                pl.split.as<uint32_t>(), pl.left.as<uint32_t>(), pl.right.as<uint32_t>(),
                pl.dl.as<uint8_t>(), pl.value.as<float>(), pl.lr, pl.init, out);
        }
        else
        {
            node_predict_kernel<uint16_t><<<ceil_div(n, 256), 256, 0, s>>>(
                static_cast<uint16_t const *>(p.bins), p.n_pad, n, pl.last.as<uint32_t>(),
                n_trees, pl.roots.as<uint32_t>(), pl.feature.as<uint32_t>(),
                pl.split.as<uint32_t>(), pl.left.as<uint32_t>(), pl.right.as<uint32_t>(),
                pl.dl.as<uint8_t>(), pl.value.as<float>(), pl.lr, pl.init, out);
        }
        BB_LAUNCH("node_predict_kernel");
        return 1;
    }
    if (pl.depth <= k_lane_depth)
    {
        auto const *mirror = static_cast<uint32_t const *>(p.mirror);
        if (n <= k_few_rows)
        {
            auto const fn = pl.u8 ? few_values_kernel<uint8_t> : few_values_kernel<uint16_t>;
            fn<<<dim3(static_cast<uint32_t>(n), ceil_div(n_trees, k_few_threads)), k_few_threads, 0,
                 s>>>(mirror, n, pl.n_tiles, pl.last_words,
                      pl.heaps, pl.depth, n_trees, pl.few_vals);
            BB_LAUNCH("few_values_kernel");
            launch_k(true, few_sum_kernel, static_cast<uint32_t>(n), k_few_threads, 0, s,
                     pl.few_vals, n_trees, pl.lr, pl.init, out);
            BB_LAUNCH("few_sum_kernel");
            return 2;
        }
        if (row_form(n, n_trees, pl.sms))
        {
            uint32_t const T = std::min(row_threads(n, pl.sms), ((n_trees + 31) / 32) * 32);
            auto const     fn = pl.u8 ? row_predict_kernel<uint8_t> : row_predict_kernel<uint16_t>;
            fn<<<static_cast<uint32_t>(n), T, 0, s>>>(mirror, n, pl.n_tiles,
                                                      pl.last_words,
                                                      pl.heaps, pl.depth, n_trees,
                                                      pl.lr, pl.init, out);
            BB_LAUNCH("row_predict_kernel");
            return 1;
        }
        if (pl.heap_ctas != 0 && by_row(pl, n, n_trees))
        {
            return heap_launch(pl, p, n_trees, out, s);
        }
        // equal tiles, in as few waves of two CTAs an SM as the largest allows
        uint64_t const wave  = uint64_t{2} * pl.sms;
        uint64_t const waves = (n + (wave * pl.lane_rows) - 1) / (wave * pl.lane_rows);
        uint32_t const rows  = ceil_div(n, wave * waves);
        lane_fn(pl.u8, pl.depth)<<<ceil_div(n, rows), k_lane_threads,
                                   lane_smem(pl.depth, pl.n_tiles, rows), s>>>(
            mirror, n, pl.n_tiles, pl.last_words, pl.heaps, n_trees,
            rows, pl.lr, pl.init, out);
        BB_LAUNCH("lane_predict_kernel");
        return 1;
    }
    if (ceil_div(n, 256) < pl.sms && n * static_cast<size_t>(n_trees) * sizeof(float) <= k_max_vals)
    {
        return split_launch(pl, p, n_trees, out, s);
    }
    return heap_launch(pl, p, n_trees, out, s);
}

std::unique_ptr<bb_predict_plan> make_plan(Plane const &p, uint32_t n_trees,
                                           uint32_t const *roots, uint32_t n_nodes,
                                           uint32_t const *feature, uint32_t const *split_bin,
                                           uint32_t const *left, uint32_t const *right,
                                           uint8_t const *default_left, float const *value,
                                           float lr, float init)
{
    need(roots != nullptr && feature != nullptr && split_bin != nullptr && left != nullptr &&
             right != nullptr && default_left != nullptr && value != nullptr,
         "bb_predict_plan_create: null argument");
    need(n_trees > 0 && n_nodes > 0, "bb_predict_plan_create: empty ensemble");
    validate_trees(p, n_trees, roots, n_nodes, feature, left, right);
    auto pl     = std::make_unique<bb_predict_plan>();
    pl->n_feats = p.n_feats;
    pl->u8      = p.u8;
    pl->cut_off.assign(p.h_cut_off, p.h_cut_off + p.n_feats + 1);
    pl->n_trees = n_trees;
    pl->lr      = lr;
    pl->init    = init;
    uint32_t D  = 1;
    for (uint32_t t = 0; t < n_trees; ++t)
    {
        uint32_t const e = t + 1 < n_trees ? roots[t + 1] : n_nodes;
        D = std::max(D, tree_depth(roots[t], e, feature, left, right));
    }
    uint32_t const per     = k_mirror_bytes / (p.u8 ? 1u : 2u);
    uint32_t const n_tiles = (p.n_feats + per - 1) / per;
    if (D <= k_max_heap_depth && n_tiles <= k_max_heap_tiles && p.mirror != nullptr)
    {
        pl->depth          = D;
        pl->n_tiles        = n_tiles;
        size_t const   slots = static_cast<size_t>(2u << D);
        uint32_t const words = n_tiles * 8;
        bool const       by_tree = D <= k_lane_depth;
        HeapPacker const pk{D,       p.u8,      words, by_tree, by_tree ? 32u : 1u, pl->cut_off.data(),
                            feature, split_bin, left,  right,   default_left,       value};
        pl->sms = sm_count();
        // the heaps, then the last words
        size_t const          n_heap = slots * (by_tree ? 32 * ((n_trees + 31) / 32) : n_trees);
        std::vector<uint32_t> h(n_heap + words, by_tree ? pk.never() : 0u);
        for (uint32_t t = 0; t < n_trees; ++t)
        {
            // 32 trees interleaved (the last group's missing ones, never added, route
            // every row to their left spine), or one after another
            size_t const at = by_tree ? ((t / 32) * slots * 32) + (t % 32) : t * slots;
            pk.fill(h.data() + at, roots[t], roots[t], 1, 0);
        }
        if (by_tree)
        {
            size_t const per_row = lane_smem(D, n_tiles, 1) - lane_smem(D, n_tiles, 0);
            pl->lane_rows        = static_cast<uint32_t>(std::min<size_t>(
                k_lane_threads, (k_lane_smem - lane_smem(D, n_tiles, 0)) / per_row));
            allow_smem(lane_fn(p.u8, D));
        }
        if (D > k_lane_depth || n_tiles <= 2)
        {
            uint32_t const T  = heap_threads(D, n_tiles);
            HeapFn const   fn = heap_fn(p.u8, D, T);
            allow_smem(fn);
            if (D > k_lane_depth)
            {
                allow_smem(heap_fn(p.u8, D, 256));
            }
            int occ = 0;
            check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, static_cast<int>(T),
                                                                heap_smem(D, n_tiles, T)),
                  "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
            pl->heap_ctas = static_cast<uint64_t>(std::max(occ, 1)) * pl->sms;
        }
        // the last bin of every code lane of every staged word (padding
        // lanes: a value no code has)
        uint32_t const lanes = p.u8 ? 4u : 2u;
        for (uint32_t wd = 0; wd < words; ++wd)
        {
            uint32_t v = 0;
            for (uint32_t k = 0; k < lanes; ++k)
            {
                uint32_t const f    = (wd * lanes) + k;
                uint32_t const last = f < p.n_feats ? p.h_cut_off[f + 1] - p.h_cut_off[f] - 1
                                                    : (p.u8 ? 0xFFu : 0xFFFFu);
                v |= last << (k * (32u / lanes));
            }
            h[n_heap + wd] = v;
        }
        size_t const n_few = by_tree ? size_t{k_few_rows} * n_trees : 0;
        pl->tables.alloc((h.size() + n_few) * 4);
        pl->heaps      = pl->tables.as<uint32_t>();
        pl->last_words = pl->heaps + n_heap;
        pl->few_vals   = reinterpret_cast<float *>(pl->last_words + words);
        check(cudaMemcpy(pl->heaps, h.data(), h.size() * 4, cudaMemcpyHostToDevice), "cudaMemcpy");
    }
    else
    {
        std::vector<uint32_t> last(p.n_feats);
        for (uint32_t f = 0; f < p.n_feats; ++f)
        {
            last[f] = p.h_cut_off[f + 1] - p.h_cut_off[f] - 1;
        }
        pl->last.upload(last.data(), p.n_feats * 4ull);
        pl->roots.upload(roots, n_trees * 4ull);
        pl->feature.upload(feature, n_nodes * 4ull);
        pl->split.upload(split_bin, n_nodes * 4ull);
        pl->left.upload(left, n_nodes * 4ull);
        pl->right.upload(right, n_nodes * 4ull);
        pl->dl.upload(default_left, n_nodes);
        pl->value.upload(value, n_nodes * 4ull);
    }
    check(cudaStreamCreateWithFlags(&pl->stream, cudaStreamNonBlocking), "cudaStreamCreate");
    return pl;
}

void plan_run_host(bb_predict_plan &pl, Plane const &p, uint32_t n_trees, float *out)
{
    std::lock_guard<std::mutex> lock(pl.mu);
    size_t const bytes = p.n_rows * sizeof(float);
    if (bytes == 0)
    {
        return;
    }
    if (pl.out_cap < bytes)
    {
        if (pl.out != nullptr)
        {
            check(cudaFree(pl.out), "cudaFree");
            pl.out     = nullptr;
            pl.out_cap = 0;
        }
        check(cudaMalloc(&pl.out, bytes), "cudaMalloc");
        pl.out_cap = bytes;
    }
    plan_launch(pl, p, n_trees, pl.out, pl.stream);
    check(cudaMemcpyAsync(out, pl.out, bytes, cudaMemcpyDeviceToHost, pl.stream),
          "cudaMemcpyAsync");
    check(cudaStreamSynchronize(pl.stream), "cudaStreamSynchronize");
}

uint32_t trees_to_run(bb_predict_plan const &pl, uint32_t n_trees)
{
    need(n_trees <= pl.n_trees, "bb_predict_plan: more trees asked than the plan holds");
    return n_trees == 0 ? pl.n_trees : n_trees;
}

} // namespace
} // namespace bb

using namespace bb;

extern "C"
{
    int bb_predict_plan_create(bb_plane const *plane, uint32_t n_trees, uint32_t const *roots,
                               uint32_t n_nodes, uint32_t const *feature,
                               uint32_t const *split_bin, uint32_t const *left,
                               uint32_t const *right, uint8_t const *default_left,
                               float const *value, float lr, float init, bb_predict_plan **out)
    {
        return guarded(
            [&]
            {
                need(plane != nullptr && out != nullptr, "bb_predict_plan_create: null argument");
                *out = make_plan(plane->p, n_trees, roots, n_nodes, feature, split_bin, left,
                                 right, default_left, value, lr, init)
                           .release();
            });
    }

    int bb_predict_plan_run(bb_predict_plan *plan, bb_plane const *plane, uint32_t n_trees,
                            float *out)
    {
        return guarded(
            [&]
            {
                need(plan != nullptr && plane != nullptr && out != nullptr,
                     "bb_predict_plan_run: null argument");
                plan_check_plane(*plan, plane->p);
                plan_run_host(*plan, plane->p, trees_to_run(*plan, n_trees), out);
            });
    }

    int bb_predict_plan_launch(bb_predict_plan *plan, bb_plane const *plane, uint32_t n_trees,
                               float *out_device, void *stream, uint32_t *launches)
    {
        return guarded(
            [&]
            {
                need(plan != nullptr && plane != nullptr && out_device != nullptr,
                     "bb_predict_plan_launch: null argument");
                plan_check_plane(*plan, plane->p);
                std::lock_guard<std::mutex> lock(plan->mu);
                uint32_t const k = plan_launch(*plan, plane->p, trees_to_run(*plan, n_trees),
                                               out_device, static_cast<cudaStream_t>(stream));
                if (launches != nullptr)
                {
                    *launches = k;
                }
            });
    }

    int bb_predict_plan_depth(bb_predict_plan const *plan, uint32_t *depth)
    {
        return guarded(
            [&]
            {
                need(plan != nullptr && depth != nullptr, "bb_predict_plan_depth: null argument");
                *depth = plan->depth;
            });
    }

    void bb_predict_plan_destroy(bb_predict_plan *plan)
    {
        delete plan;
    }

    int bb_predict(bb_plane const *plane, uint32_t n_trees, uint32_t const *roots,
                   uint32_t n_nodes, uint32_t const *feature, uint32_t const *split_bin,
                   uint32_t const *left, uint32_t const *right, uint8_t const *default_left,
                   float const *value, float lr, float init, float *out)
    {
        return guarded(
            [&]
            {
                need(plane != nullptr && out != nullptr, "bb_predict: null argument");
                auto pl = make_plan(plane->p, n_trees, roots, n_nodes, feature, split_bin, left,
                                    right, default_left, value, lr, init);
                plan_run_host(*pl, plane->p, n_trees, out);
            });
    }
}
