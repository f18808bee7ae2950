#include "ingest.cuh"

#include <algorithm>
#include <vector>

namespace bb
{
namespace
{

constexpr uint32_t k_tile_rows  = 256; // rows per CTA tile
constexpr uint32_t k_tile_feats = 32;  // features per CTA tile
constexpr uint32_t k_threads    = 256;
constexpr uint32_t k_bin_ctas   = 148 * 2; // two CTAs' padded tables and tiles fit an SM
constexpr size_t   k_max_smem   = 227 * 1024;
// Batches of up to this many values (whole tiles of features counted) take a
// thread per value. It writes single bytes to columns far apart and reads its cuts
// from L2, so what it costs goes with the values, where a wave of row tiles takes
// about 20 us whatever is in it. Refills from device memory, wall us by value / by
// row tiles, 255 cuts: 8,000 x 28 26.4 / 33.4, 16,000 x 28 31.5 / 33.8; 1,000 x
// 333 32.7 / 34.8, 2,000 x 333 40.4 / 36.6; 250 x 1,000 30.0 / 35.7, 500 x 1,000
// 36.7 / 34.0, 8,000 x 1,000 260 / 99.
constexpr uint64_t k_small_values = 3 << 17;
constexpr uint32_t k_pad_cuts   = 256;

// lower_bound for K values over K tables of cuts at once (cut(k, i) is table
// k's cut i, nb[k] of them): pos[k] = the number of cuts below x[k]. A step
// halves what is left of every table, whatever the values, so the K chains of
// dependent loads overlap.
template <uint32_t K, typename Load>
__device__ __forceinline__ void lower_bounds(Load const &cut, uint32_t const (&nb)[K],
                                             float const (&x)[K], uint32_t (&pos)[K])
{
    uint32_t n[K];
    uint32_t most = 0;
#pragma unroll
    for (uint32_t k = 0; k < K; ++k)
    {
        pos[k] = 0;
        n[k]   = nb[k];
        most   = max(most, nb[k]);
    }
    for (; most > 1; most -= most >> 1)
    {
#pragma unroll
        for (uint32_t k = 0; k < K; ++k)
        {
            uint32_t const half = n[k] >> 1;
            if (half != 0)
            {
                pos[k] += cut(k, pos[k] + half - 1) < x[k] ? half : 0;
            }
            n[k] -= half;
        }
    }
#pragma unroll
    for (uint32_t k = 0; k < K; ++k)
    {
        if (n[k] != 0)
        {
            pos[k] += cut(k, pos[k]) < x[k] ? 1 : 0;
        }
    }
}

// Bins of K features of a row, x their values, into the row's code words.
// PAD: feature f's table fills k_pad_cuts entries of c_s.
template <typename BinT, bool PAD, uint32_t K>
__device__ __forceinline__ void bin_features(float const *c_s, uint32_t const *coff_s,
                                             uint32_t f, uint32_t nf, float const (&x)[K],
                                             uint32_t (&code)[k_tile_feats * sizeof(BinT) / 4])
{
    constexpr uint32_t in = 4 / sizeof(BinT);
    uint32_t           pos[K];
    if constexpr (PAD)
    {
        float const *c = c_s + (f * k_pad_cuts);
#pragma unroll
        for (uint32_t q = 0; q < K; ++q)
        {
            pos[q] = 0;
        }
#pragma unroll
        for (uint32_t step = k_pad_cuts / 2; step > 0; step /= 2)
        {
#pragma unroll
            for (uint32_t q = 0; q < K; ++q)
            {
                if (c[(q * k_pad_cuts) + pos[q] + step - 1] < x[q])
                {
                    pos[q] += step;
                }
            }
        }
    }
    else
    {
        uint32_t at[K], nb[K];
#pragma unroll
        for (uint32_t q = 0; q < K; ++q)
        {
            uint32_t const ff = min(f + q, nf - 1);
            at[q]             = coff_s[ff];
            nb[q]             = coff_s[ff + 1] - at[q];
        }
        lower_bounds<K>([&](uint32_t k, uint32_t i) { return c_s[at[k] + i]; }, nb, x, pos);
    }
#pragma unroll
    for (uint32_t q = 0; q < K; ++q)
    {
        if (f + q < nf)
        {
            uint32_t const b =
                isnan(x[q]) ? coff_s[f + q + 1] - coff_s[f + q] - 1 : pos[q];
            code[(f + q) / in] |= b << (((f + q) % in) * (32 / in));
        }
    }
}

// grid: (CTAs over row tiles, ceil(F / 32)); block 256. A thread bins one row
// of a 256-row tile, eight features at a time, and owns the row's mirror
// tile(s), which leave its registers whole; the columns leave through shared
// memory as 16-byte runs of rows. A CTA keeps its features' cuts over all its
// row tiles and has the next tile's values on their way (cp.async) while it
// searches, where its shared memory holds two (TWO). PAD: every table of at most k_pad_cuts cuts, each filled up to
// that many with +inf, so that the search is eight steps of a load at a
// constant offset, a compare and a conditional add (3 instructions a step;
// tables of any length take about 20). (A thread per 16 rows of a feature,
// values one after another, the cuts staged again for every tile, and a second
// pass for the mirror: 238 us for a 1M x 28 refill from device memory, 177
// so.)
constexpr uint32_t k_x_stride = k_tile_feats + 4; // floats: rows' 16-byte quarters in
                                                  // different banks

template <typename BinT, bool PAD, bool TWO>
__global__ void __launch_bounds__(k_threads, 2)
    bin_apply_kernel(float const *__restrict__ X, uint64_t n_rows, uint32_t F,
                     uint64_t row0, float const *__restrict__ cuts,
                     uint32_t const *__restrict__ cut_off, BinT *__restrict__ bins,
                     uint64_t n_pad, uint4 *__restrict__ mirror, uint64_t m_rows,
                     uint32_t max_tile_cuts, bool vec4)
{
    extern __shared__ __align__(16) float smem[];
    constexpr uint32_t x_floats = k_tile_rows * k_x_stride;
    float             *c_s      = smem + ((TWO ? 2 : 1) * x_floats);
    uint32_t          *coff_s   = reinterpret_cast<uint32_t *>(c_s + max_tile_cuts);
    constexpr uint32_t per      = 16 / sizeof(BinT);
    constexpr uint32_t words    = k_tile_feats * sizeof(BinT) / 4; // of a row's codes
    constexpr uint32_t in       = 4 / sizeof(BinT);

    uint32_t const f0 = blockIdx.y * k_tile_feats;
    uint32_t const nf = min(k_tile_feats, F - f0);
    // the tile of X from row r0: features f0..f0+nf into buffer b
    auto const load = [&](uint64_t r0, uint32_t b)
    {
        if (r0 < n_rows)
        {
            uint32_t const nr =
                static_cast<uint32_t>(n_rows - r0 < k_tile_rows ? n_rows - r0 : k_tile_rows);
            float      *tile = smem + (b * x_floats);
            float const *src = X + (r0 * F) + f0;
            if (vec4)
            {
                uint32_t const q = nf / 4; // 16 bytes at a time
                for (uint32_t i = threadIdx.x; i < nr * q; i += k_threads)
                {
                    uint32_t const rr = i / q;
                    uint32_t const qq = i - (rr * q);
                    uint32_t const d  = static_cast<uint32_t>(
                        __cvta_generic_to_shared(tile + (rr * k_x_stride) + (qq * 4)));
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d),
                                 "l"(src + (static_cast<uint64_t>(rr) * F) + (qq * 4)));
                }
            }
            else
            {
                for (uint32_t i = threadIdx.x; i < nr * nf; i += k_threads)
                {
                    uint32_t const rr = i / nf;
                    uint32_t const ff = i - (rr * nf);
                    uint32_t const d  = static_cast<uint32_t>(
                        __cvta_generic_to_shared(tile + (rr * k_x_stride) + ff));
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d),
                                 "l"(src + (static_cast<uint64_t>(rr) * F) + ff));
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    uint64_t const stride = static_cast<uint64_t>(gridDim.x) * k_tile_rows;
    uint64_t       r0     = static_cast<uint64_t>(blockIdx.x) * k_tile_rows;
    load(r0, 0);
    // the features' cuts
    if (threadIdx.x <= nf)
    {
        coff_s[threadIdx.x] = cut_off[f0 + threadIdx.x] - cut_off[f0];
    }
    uint32_t const c_begin = cut_off[f0];
    if constexpr (PAD)
    {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < k_tile_feats * k_pad_cuts; i += k_threads)
        {
            uint32_t const ff = i / k_pad_cuts;
            uint32_t const k  = i % k_pad_cuts;
            c_s[i] = ff < nf && k < coff_s[ff + 1] - coff_s[ff] ? cuts[c_begin + coff_s[ff] + k]
                                                                : INFINITY;
        }
    }
    else
    {
        uint32_t const c_count = cut_off[f0 + nf] - c_begin;
        for (uint32_t i = threadIdx.x; i < c_count; i += k_threads)
        {
            c_s[i] = cuts[c_begin + i];
        }
    }
    for (uint32_t b = 0; r0 < n_rows; r0 += stride, b ^= TWO ? 1 : 0)
    {
        uint32_t const nr =
            static_cast<uint32_t>(n_rows - r0 < k_tile_rows ? n_rows - r0 : k_tile_rows);
        if constexpr (TWO)
        {
            load(r0 + stride, b ^ 1);
            asm volatile("cp.async.wait_group 1;\n" ::);
        }
        else
        {
            asm volatile("cp.async.wait_all;\n" ::);
        }
        __syncthreads(); // the tile is here (and the cuts)
        float         *tile = smem + (b * x_floats);
        uint32_t const rr   = threadIdx.x;
        uint32_t       code[words];
#pragma unroll
        for (uint32_t w = 0; w < words; ++w)
        {
            code[w] = 0;
        }
        if (rr < nr)
        {
            // (values past the tile's features are whatever lies there: their
            // bins are dropped)
            auto const *mine = reinterpret_cast<float4 const *>(tile + (rr * k_x_stride));
#pragma unroll
            for (uint32_t g = 0; g < k_tile_feats / 8; ++g)
            {
                if (8 * g + 4 < nf) // uniform
                {
                    float4 const u    = mine[2 * g];
                    float4 const v    = mine[(2 * g) + 1];
                    float const  x[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
                    bin_features<BinT, PAD, 8>(c_s, coff_s, 8 * g, nf, x, code);
                }
                else if (8 * g < nf)
                {
                    float4 const u    = mine[2 * g];
                    float const  x[4] = {u.x, u.y, u.z, u.w};
                    bin_features<BinT, PAD, 4>(c_s, coff_s, 8 * g, nf, x, code);
                }
            }
        }
        __syncthreads(); // every row's values are taken: the columns in their place
        auto *col = reinterpret_cast<BinT *>(tile); // [feature][rows]
#pragma unroll
        for (uint32_t ff = 0; ff < k_tile_feats; ++ff)
        {
            if (ff < nf)
            {
                col[(ff * k_tile_rows) + rr] =
                    static_cast<BinT>(code[ff / in] >> ((ff % in) * (32 / in)));
            }
        }
        if (rr < nr && mirror != nullptr)
        {
            // a tile of 32 bytes (u8), or two of them (u16)
#pragma unroll
            for (uint32_t t = 0; t < words / 8; ++t)
            {
                uint32_t const at = (blockIdx.y * (words / 8)) + t;
                if (t == 0 || nf > t * (k_mirror_bytes / sizeof(BinT)))
                {
                    uint4 *m =
                        mirror + (((static_cast<uint64_t>(at) * m_rows) + row0 + r0 + rr) * 2);
                    m[0] = make_uint4(code[8 * t], code[(8 * t) + 1], code[(8 * t) + 2],
                                      code[(8 * t) + 3]);
                    m[1] = make_uint4(code[(8 * t) + 4], code[(8 * t) + 5], code[(8 * t) + 6],
                                      code[(8 * t) + 7]);
                }
            }
        }
        __syncthreads();
        // one 16-byte store per (feature, run of rows)
        constexpr uint32_t runs = k_tile_rows / per;
        for (uint32_t i = threadIdx.x; i < nf * runs; i += k_threads)
        {
            uint32_t const ff = i / runs;
            uint32_t const rb = (i % runs) * per;
            if (rb < nr)
            {
                BinT *dst = bins + (static_cast<uint64_t>(f0 + ff) * n_pad) + row0 + r0 + rb;
                *reinterpret_cast<uint4 *>(dst) =
                    *reinterpret_cast<uint4 const *>(col + (ff * k_tile_rows) + rb);
            }
        }
        __syncthreads(); // the columns have left: the buffer may be filled again
        if constexpr (!TWO)
        {
            load(r0 + stride, 0);
        }
    }
    asm volatile("cp.async.wait_all;\n" ::);
}

// Small batches: a thread per (row, feature slot), the cuts from L2, a byte
// (or two) into the column and into the mirror. No tile's cuts to stage: a
// request of one row took 9 us of that.
template <typename BinT>
__global__ void __launch_bounds__(k_threads)
    bin_rows_kernel(float const *__restrict__ X, uint64_t n_rows, uint32_t F, uint64_t row0,
                    float const *__restrict__ cuts, uint32_t const *__restrict__ cut_off,
                    BinT *__restrict__ bins, uint64_t n_pad, BinT *__restrict__ mirror,
                    uint64_t m_rows, uint32_t slots)
{
    uint64_t const i = (static_cast<uint64_t>(blockIdx.x) * k_threads) + threadIdx.x;
    uint64_t const r = i / slots;
    uint32_t const f = static_cast<uint32_t>(i - (r * slots));
    if (r >= n_rows)
    {
        return;
    }
    uint32_t b = 0; // (a slot past the features holds 0)
    if (f < F)
    {
        float const   *c     = cuts + __ldg(cut_off + f);
        uint32_t const nb[1] = {__ldg(cut_off + f + 1) - __ldg(cut_off + f)};
        float const    x[1]  = {X[(r * F) + f]};
        uint32_t       pos[1];
        lower_bounds<1>([&](uint32_t, uint32_t k) { return __ldg(c + k); }, nb, x, pos);
        b = isnan(x[0]) ? nb[0] - 1 : pos[0];
        bins[(static_cast<uint64_t>(f) * n_pad) + row0 + r] = static_cast<BinT>(b);
    }
    constexpr uint32_t per = k_mirror_bytes / sizeof(BinT);
    if (mirror != nullptr)
    {
        mirror[((((f / per) * m_rows) + row0 + r) * per) + (f % per)] = static_cast<BinT>(b);
    }
}

// One thread per (row, tile): gathers the tile's codes from the
// feature-major columns (coalesced across the warp's consecutive rows) and
// writes the row's 32-byte tile as two 16-byte stores.
template <typename BinT>
__global__ void __launch_bounds__(k_threads)
    mirror_kernel(BinT const *__restrict__ bins, uint64_t n_rows, uint64_t n_pad,
                  uint32_t F, uint4 *__restrict__ mirror)
{
    constexpr uint32_t per = k_mirror_bytes / sizeof(BinT);
    uint64_t const     r   = (static_cast<uint64_t>(blockIdx.x) * k_threads) + threadIdx.x;
    uint32_t const     t   = blockIdx.y;
    if (r >= n_rows)
    {
        return;
    }
    alignas(16) BinT v[per];
#pragma unroll
    for (uint32_t k = 0; k < per; ++k)
    {
        uint32_t const f = (t * per) + k;
        v[k]             = f < F ? bins[(static_cast<uint64_t>(f) * n_pad) + r] : BinT{0};
    }
    uint4 const   *src = reinterpret_cast<uint4 const *>(v);
    uint64_t const o   = ((static_cast<uint64_t>(t) * n_rows) + r) * 2;
    mirror[o]          = src[0];
    mirror[o + 1]      = src[1];
}

} // namespace

void alloc_codes(Plane &p, uint64_t rows)
{
    uint32_t const per   = k_mirror_bytes / (p.u8 ? 1 : 2);
    p.n_tiles            = (p.n_feats + per - 1) / per;
    uint64_t const pad   = ((rows + 63) / 64) * 64;
    size_t const   codes = ((static_cast<size_t>(p.n_feats) * pad * (p.u8 ? 1 : 2)) + 255) &
                         ~size_t{255};
    size_t const bytes   = codes + (static_cast<size_t>(p.n_tiles) * rows * k_mirror_bytes);
    MemPool::with_trim([&] { return cudaMalloc(&p.bins, bytes); }, "cudaMalloc");
    p.mirror = static_cast<char *>(p.bins) + codes;
}

void build_mirror(Plane &p, cudaStream_t stream)
{
    dim3 const grid(ceil_div(p.n_rows, k_threads), p.n_tiles);
    if (p.u8)
    {
        mirror_kernel<uint8_t><<<grid, k_threads, 0, stream>>>(
            static_cast<uint8_t const *>(p.bins), p.n_rows, p.n_pad, p.n_feats,
            static_cast<uint4 *>(p.mirror));
    }
    else
    {
        mirror_kernel<uint16_t><<<grid, k_threads, 0, stream>>>(
            static_cast<uint16_t const *>(p.bins), p.n_rows, p.n_pad, p.n_feats,
            static_cast<uint4 *>(p.mirror));
    }
    BB_LAUNCH("mirror_kernel");
}

uint64_t stage_rows_for(uint32_t n_feats, uint64_t max_rows)
{
    // at most 64 MB; when a batch can take more than one chunk, every chunk
    // starts on a tile boundary (the kernel's 16-byte code stores need the
    // chunk's first row aligned)
    uint64_t const row_bytes = static_cast<uint64_t>(n_feats) * sizeof(float);
    uint64_t       rows      = std::min<uint64_t>(max_rows, (64ull << 20) / row_bytes);
    if (rows < max_rows)
    {
        rows = std::max<uint64_t>(k_tile_rows, rows - (rows % k_tile_rows));
    }
    return std::max<uint64_t>(rows, 1);
}

void ingest(Plane &p, float const *X, bool x_on_device, cudaStream_t stream, float *owned_stage,
            uint64_t owned_rows)
{
    uint32_t const F = p.n_feats;
    // the largest per-tile cut table
    uint32_t max_tile_cuts = 0;
    for (uint32_t f0 = 0; f0 < F; f0 += k_tile_feats)
    {
        uint32_t const f1 = std::min(F, f0 + k_tile_feats);
        max_tile_cuts     = std::max(max_tile_cuts, p.h_cut_off[f1] - p.h_cut_off[f0]);
    }
    bool pad = true;
    for (uint32_t f = 0; f < F; ++f)
    {
        pad = pad && p.h_cut_off[f + 1] - p.h_cut_off[f] <= k_pad_cuts;
    }
    if (pad)
    {
        max_tile_cuts = k_tile_feats * k_pad_cuts;
    }
    size_t const one   = k_tile_rows * k_x_stride * sizeof(float); // a tile of values
    size_t const table = (max_tile_cuts * sizeof(float)) + ((k_tile_feats + 1) * sizeof(uint32_t));
    // (a tile of values, rows 33 apart, beside the cuts is what the capacity stands for)
    if ((k_tile_rows * (k_tile_feats + 1) * sizeof(float)) + table > k_max_smem)
    {
        throw ConfigError("ingest: a 32-feature tile's cuts exceed shared memory");
    }
    bool const   two_tiles = (2 * one) + table <= k_max_smem;
    bool const   by_value  = one + table > k_max_smem;
    size_t const smem      = ((two_tiles ? 2 : 1) * one) + table;
    // (u8 codes have at most 256 cuts a feature: padded tables, two tiles)
    auto const kern8  = bin_apply_kernel<uint8_t, true, true>;
    auto const kern16 = pad         ? bin_apply_kernel<uint16_t, true, true>
                        : two_tiles ? bin_apply_kernel<uint16_t, false, true>
                                    : bin_apply_kernel<uint16_t, false, false>;
    if (!by_value)
    {
        p.u8 ? allow_smem(kern8) : allow_smem(kern16);
    }
    bool const vec4 = (F % 4) == 0 &&
                      (!x_on_device || (reinterpret_cast<uintptr_t>(X) % 16) == 0);

    auto launch = [&](float const *Xd, uint64_t rows, uint64_t row0)
    {
        uint32_t const per   = k_mirror_bytes / (p.u8 ? 1 : 2);
        uint32_t const slots = p.n_tiles * per;
        if (rows * slots <= k_small_values || by_value)
        {
            uint32_t const grid  = ceil_div(rows * slots, k_threads);
            if (p.u8)
            {
                bin_rows_kernel<uint8_t><<<grid, k_threads, 0, stream>>>(
                    Xd, rows, F, row0, p.cuts, p.cut_off, static_cast<uint8_t *>(p.bins), p.n_pad,
                    static_cast<uint8_t *>(p.mirror), p.n_rows, slots);
            }
            else
            {
                bin_rows_kernel<uint16_t><<<grid, k_threads, 0, stream>>>(
                    Xd, rows, F, row0, p.cuts, p.cut_off, static_cast<uint16_t *>(p.bins), p.n_pad,
                    static_cast<uint16_t *>(p.mirror), p.n_rows, slots);
            }
            BB_LAUNCH("bin_rows_kernel");
            return;
        }
        // a CTA keeps its features' cuts over its row tiles: no more CTAs than about
        // fit the GPU at once (one more than fit takes as long again: 333 features
        // as 27 x 11 CTAs, of which 296 fit, 54.0 us for 8,000 rows, as 26 x 11 50.1)
        uint32_t const ftiles = ceil_div(F, k_tile_feats);
        dim3 const     grid(std::min(ceil_div(rows, k_tile_rows), std::max(1u, k_bin_ctas / ftiles)),
                            ftiles);
        if (p.u8)
        {
            kern8<<<grid, k_threads, smem, stream>>>(
                Xd, rows, F, row0, p.cuts, p.cut_off, static_cast<uint8_t *>(p.bins), p.n_pad,
                static_cast<uint4 *>(p.mirror), p.n_rows, max_tile_cuts, vec4);
        }
        else
        {
            kern16<<<grid, k_threads, smem, stream>>>(
                Xd, rows, F, row0, p.cuts, p.cut_off, static_cast<uint16_t *>(p.bins), p.n_pad,
                static_cast<uint4 *>(p.mirror), p.n_rows, max_tile_cuts, vec4);
        }
        BB_LAUNCH("bin_apply_kernel");
    };

    if (x_on_device)
    {
        launch(X, p.n_rows, 0);
        return;
    }
    if (owned_stage != nullptr)
    {
        if (owned_rows < p.n_rows && owned_rows % k_tile_rows != 0)
        {
            throw std::logic_error("ingest: a staging buffer that chunks must hold whole tiles");
        }
        // a request plane: one staging buffer the plane owns, copy then bin
        // chunk by chunk on the one stream (no allocation)
        uint64_t const row_bytes = static_cast<uint64_t>(F) * sizeof(float);
        for (uint64_t r0 = 0; r0 < p.n_rows; r0 += owned_rows)
        {
            uint64_t const rows = std::min(owned_rows, p.n_rows - r0);
            BB_CHECK(cudaMemcpyAsync(owned_stage, X + (r0 * F), rows * row_bytes,
                                     cudaMemcpyHostToDevice, stream));
            launch(owned_stage, rows, r0);
        }
        return;
    }
    // Host input: stream it through two device staging buffers of <= 64 MB
    // (a multiple of the tile rows), copy of chunk k+1 overlapping the bin
    // kernel of chunk k.
    uint64_t const row_bytes  = static_cast<uint64_t>(F) * sizeof(float);
    uint64_t       chunk_rows = std::max<uint64_t>(k_tile_rows, (64ull << 20) / row_bytes);
    chunk_rows -= chunk_rows % k_tile_rows;
    chunk_rows = std::min<uint64_t>(chunk_rows, ((p.n_rows + k_tile_rows - 1) / k_tile_rows) *
                                                    k_tile_rows);
    float      *stage[2] = {nullptr, nullptr};
    cudaEvent_t done[2];
    cudaStream_t copy_s;
    BB_CHECK(cudaStreamCreateWithFlags(&copy_s, cudaStreamNonBlocking));
    for (int i = 0; i < 2; ++i)
    {
        BB_CHECK(cudaMallocAsync(&stage[i], chunk_rows * row_bytes, stream));
        BB_CHECK(cudaEventCreateWithFlags(&done[i], cudaEventDisableTiming));
        BB_CHECK(cudaEventRecord(done[i], stream));
    }
    cudaEvent_t copied;
    BB_CHECK(cudaEventCreateWithFlags(&copied, cudaEventDisableTiming));
    int k = 0;
    for (uint64_t r0 = 0; r0 < p.n_rows; r0 += chunk_rows, k ^= 1)
    {
        uint64_t const rows = std::min(chunk_rows, p.n_rows - r0);
        BB_CHECK(cudaStreamWaitEvent(copy_s, done[k], 0));
        BB_CHECK(cudaMemcpyAsync(stage[k], X + (r0 * F), rows * row_bytes,
                                 cudaMemcpyHostToDevice, copy_s));
        BB_CHECK(cudaEventRecord(copied, copy_s));
        BB_CHECK(cudaStreamWaitEvent(stream, copied, 0));
        launch(stage[k], rows, r0);
        BB_CHECK(cudaEventRecord(done[k], stream));
    }
    for (int i = 0; i < 2; ++i)
    {
        BB_CHECK(cudaFreeAsync(stage[i], stream));
        BB_CHECK(cudaEventDestroy(done[i]));
    }
    BB_CHECK(cudaEventDestroy(copied));
    BB_CHECK(cudaStreamSynchronize(stream));
    BB_CHECK(cudaStreamDestroy(copy_s));
}

} // namespace bb
