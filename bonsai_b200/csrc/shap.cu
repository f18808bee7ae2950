// Device TreeSHAP (bb_pred_contribs): per-row SHAP contributions of an
// ensemble in bin space, in FP64.
//
// The reference computes them host-side with Lundberg et al.'s Algorithm 2
// (extend/unwind over a "unique path", src/shap.cpp:20-213) and device-side
// in FP32 over packed leaf paths (src/cuda/shap.cu:63-169, packer
// src/shap_paths.cpp). This kernel uses the path form of the same quantity:
// every root-to-leaf path, with the conditions on one feature merged into a
// single element i carrying its cover fraction z_i (the product of
// cover(child) / cover(parent) over that feature's splits) and the row's
// indicator o_i (1 when the row satisfies all of them), contributes
//
//     phi[f_i] += v * (o_i - z_i) * integral_0^1 prod_{j != i} (z_j + (o_j - z_j) t) dt
//
// because the Shapley weights |S|!(n-1-|S|)!/n! are the Beta integrals
// integral t^|S| (1-t)^(n-1-|S|) dt. The integrand is a polynomial of degree
// n - 1, so an m-point Gauss-Legendre rule with 2m - 1 >= n - 1 is exact; the
// products over j != i come from prefix and suffix products, with no
// division. The bias column is the reference's expected value per tree
// (tree_expected_value, src/shap.cpp:250-290), then the booster's
// composition: phi *= lr, phi[F] += init (include/bonsai/booster.hpp:903-924).
//
// Ensembles of depth at most 8 take another form of the sum, tree by tree (the
// tree form, below). For the others, the ensemble's paths are packed once
// (bb_shap_plan_create; the reference's cuda_shap_plan,
// include/bonsai/cuda/shap.hpp:31-35) into fixed-stride records of K elements
// (K = 8, 16 or 32 by the longest path) and streamed through shared memory in chunks. A CTA covers a tile of rows crossed with
// PL path lanes: thread (row, lane) takes every PL-th path of the chunk
// against its row's codes (staged in shared memory) and accumulates into its
// own FP64 slice; with PL = 1 every thread of a warp reads the same path
// (broadcast loads, no divergence). Small batches raise PL and split the
// paths across CTAs, each split writing its partial sums; slices and splits
// are summed in a fixed order, so results are bit-identical run to run.
#include "bonsai_b200.h"
#include "ingest.cuh"

#include <algorithm>
#include <cmath>
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

constexpr uint32_t k_max_path       = 32; // merged elements per path
constexpr uint32_t k_max_gauss      = 16;
constexpr uint32_t k_max_shap_feats = 128;
constexpr uint32_t k_sms            = 148;
constexpr size_t   k_chunk_budget   = 16384;
constexpr size_t   k_max_ws_bytes   = size_t{256} << 20;

// One merged path element: the feature and whether the missing (last) bin
// passes, the non-missing bins [lo, hi] its conditions leave (lo > hi:
// none), and the product of its cover fractions.
struct PathElem
{
    uint32_t fm;   // feature | miss_ok << 31
    uint32_t lohi; // lo | hi << 16
    double   zero;
};

struct PathHead
{
    double   value;
    uint32_t count;
    uint32_t pad;
};

struct Gauss
{
    double   x[k_max_gauss];
    double   w[k_max_gauss];
    uint32_t m;
};

// Contributions of the paths [blockIdx.y * paths_per_split, + paths_per_split)
// for rows [blockIdx.x * rpb, + rpb), rpb = blockDim.x >> lane_shift. Thread
// t is row t >> lane_shift, lane t & (PL - 1). out != nullptr: the composed
// row (x lr, bias column + bias and init); else the split's raw sums into
// ws[(blockIdx.y * n_rows + r) * (F + 1) + f].
template <uint32_t K>
__global__ void __launch_bounds__(128)
    shap_tile_kernel(uint8_t const *__restrict__ bins8, uint16_t const *__restrict__ bins16,
                     uint64_t n_pad, uint64_t n_rows, uint32_t const *__restrict__ last_bin,
                     uint32_t F, PathHead const *__restrict__ heads,
                     PathElem const *__restrict__ elems, uint32_t n_paths,
                     uint32_t paths_per_split, uint32_t chunk, uint32_t lane_shift, Gauss g,
                     double lr, double bias, double init, double *__restrict__ out,
                     double *__restrict__ ws)
{
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t const T    = blockDim.x;
    uint32_t const t    = threadIdx.x;
    uint32_t const PL   = 1u << lane_shift;
    uint32_t const rpb  = T >> lane_shift;
    uint32_t const rl   = t >> lane_shift;
    uint32_t const lane = t & (PL - 1u);
    auto *const    phi_s   = reinterpret_cast<double *>(smem);             // [F + 1][T]
    auto *const    heads_s = reinterpret_cast<PathHead *>(phi_s + ((F + 1) * T));
    // path j's elements at elems_s[j * (K + 1)]: the odd stride puts the
    // paths of different lanes on different banks
    auto *const    elems_s = reinterpret_cast<PathElem *>(heads_s + chunk);
    // row rl's code of feature f at codes_s[f * (rpb + 1) + rl]: lanes of one
    // row reading different features land on different banks
    auto *const    codes_s = reinterpret_cast<uint16_t *>(elems_s + (chunk * (K + 1)));
    auto *const    last_s  = reinterpret_cast<uint32_t *>(codes_s + (((F * (rpb + 1)) + 1) & ~1u));
    uint64_t const row0 = static_cast<uint64_t>(blockIdx.x) * rpb;
    uint64_t const row  = row0 + rl;

    for (uint32_t i = t; i < F * rpb; i += T)
    {
        uint32_t const f  = i / rpb;
        uint32_t const rr = i - (f * rpb);
        uint64_t const r  = row0 + rr;
        uint32_t       c = 0;
        if (r < n_rows)
        {
            c = bins8 != nullptr ? bins8[(static_cast<uint64_t>(f) * n_pad) + r]
                                 : bins16[(static_cast<uint64_t>(f) * n_pad) + r];
        }
        codes_s[(f * (rpb + 1)) + rr] = static_cast<uint16_t>(c);
    }
    __shared__ double gx_s[k_max_gauss];
    __shared__ double gw_s[k_max_gauss];
    for (uint32_t f = t; f < F; f += T)
    {
        last_s[f] = last_bin[f];
    }
    if (t < g.m)
    {
        gx_s[t] = g.x[t];
        gw_s[t] = g.w[t];
    }
    for (uint32_t f = 0; f <= F; ++f)
    {
        phi_s[(f * T) + t] = 0.0;
    }
    uint32_t const p0 = blockIdx.y * paths_per_split;
    uint32_t const p1 = min(n_paths, p0 + paths_per_split);
    for (uint32_t c0 = p0; c0 < p1; c0 += chunk)
    {
        uint32_t const nc = min(chunk, p1 - c0);
        __syncthreads(); // the previous chunk's paths are done (and codes staged)
        {
            auto const *hs = reinterpret_cast<uint4 const *>(heads + c0);
            auto       *hd = reinterpret_cast<uint4 *>(heads_s);
            for (uint32_t i = t; i < nc; i += T)
            {
                hd[i] = hs[i];
            }
            auto const    *es = reinterpret_cast<uint4 const *>(elems + (static_cast<size_t>(c0) * K));
            auto          *ed = reinterpret_cast<uint4 *>(elems_s);
            uint32_t const ne = nc * K;
            for (uint32_t i = t; i < ne; i += T)
            {
                uint32_t const j = i / K;
                ed[i + j]        = es[i];
            }
        }
        __syncthreads();
        if (row >= n_rows)
        {
            continue;
        }
        for (uint32_t j = lane; j < nc; j += PL)
        {
            PathHead const  h = heads_s[j];
            PathElem const *e = elems_s + (j * (K + 1));
            uint32_t const  n = h.count;
            double          z[K];
            double          d[K];
            double          S[K];
            uint32_t        fe[K];
#pragma unroll
            for (uint32_t i = 0; i < K; ++i)
            {
                z[i]  = 1.0;
                d[i]  = 0.0;
                S[i]  = 0.0;
                fe[i] = 0;
                if (i < n)
                {
                    PathElem const x  = e[i];
                    uint32_t const f  = x.fm & 0x7FFFFFFFu;
                    uint32_t const bn = codes_s[(f * (rpb + 1)) + rl];
                    bool const     on = bn == last_s[f] ? (x.fm >> 31) != 0
                                                        : (bn >= (x.lohi & 0xFFFFu) &&
                                                           bn <= (x.lohi >> 16));
                    z[i]  = x.zero;
                    d[i]  = (on ? 1.0 : 0.0) - x.zero;
                    fe[i] = f;
                }
            }
            // the Gauss-Legendre points are independent chains: unrolled, a
            // thread keeps several in flight. Padded elements have factor
            // exactly 1 (z = 1, d = 0), so the products need no predicate.
            constexpr uint32_t KU = K <= 16 ? K / 2 : 1; // points per unrolled step
            for (uint32_t k0 = 0; k0 < g.m; k0 += KU)
            {
#pragma unroll
                for (uint32_t kk = 0; kk < KU; ++kk)
                {
                    uint32_t const k = k0 + kk;
                    if (k >= g.m)
                    {
                        break;
                    }
                    double const x = gx_s[k];
                    double const w = gw_s[k];
                    double       fk[K];
                    double       pre[K];
#pragma unroll
                    for (uint32_t i = 0; i < K; ++i)
                    {
                        fk[i] = __fma_rn(d[i], x, z[i]);
                    }
                    pre[0] = 1.0;
#pragma unroll
                    for (uint32_t i = 1; i < K; ++i)
                    {
                        pre[i] = pre[i - 1] * fk[i - 1];
                    }
                    double suf = 1.0;
#pragma unroll
                    for (uint32_t ii = K; ii-- > 0;)
                    {
                        S[ii] = __fma_rn(w, pre[ii] * suf, S[ii]);
                        suf *= fk[ii];
                    }
                }
            }
#pragma unroll
            for (uint32_t i = 0; i < K; ++i)
            {
                if (i < n)
                {
                    phi_s[(fe[i] * T) + t] += h.value * d[i] * S[i];
                }
            }
        }
    }
    __syncthreads();
    // a row's lanes in a fixed order, then composed or kept as the split's sum
    for (uint32_t i = t; i < rpb * (F + 1); i += T)
    {
        uint32_t const r_l = i / (F + 1);
        uint32_t const f   = i - (r_l * (F + 1));
        uint64_t const r   = row0 + r_l;
        if (r >= n_rows)
        {
            continue;
        }
        double s = 0.0;
        for (uint32_t l = 0; l < PL; ++l)
        {
            s += phi_s[(f * T) + (r_l << lane_shift) + l];
        }
        if (out != nullptr)
        {
            out[(r * (F + 1)) + f] = f == F ? ((s + bias) * lr) + init : s * lr;
        }
        else
        {
            ws[((static_cast<uint64_t>(blockIdx.y) * n_rows + r) * (F + 1)) + f] = s;
        }
    }
}

// The splits' sums in split order, composed.
__global__ void shap_reduce_kernel(double const *__restrict__ ws, uint64_t n_rows, uint32_t F,
                                   uint32_t splits, double lr, double bias, double init,
                                   double *__restrict__ out)
{
    uint64_t const i = (static_cast<uint64_t>(blockIdx.x) * blockDim.x) + threadIdx.x;
    uint64_t const n = n_rows * (F + 1);
    if (i >= n)
    {
        return;
    }
    uint32_t const f = static_cast<uint32_t>(i % (F + 1));
    double         s = 0.0;
    for (uint32_t k = 0; k < splits; ++k)
    {
        s += ws[(static_cast<uint64_t>(k) * n) + i];
    }
    out[i] = f == F ? ((s + bias) * lr) + init : s * lr;
}

// ---- the tree form ----
//
// Ensembles of depth at most 8 whose covers add up (every split node's cover
// is positive and its children's sum to it exactly: covers are row counts)
// take whole trees instead of paths. With G_k the product, at Gauss point
// t_k, of the factors z + (o - z) t_k of the path down to a node (times the
// point's weight), and A_k the sum over the leaves below it of value times
// the factors from the node down, a node of children L and R adds
//
//     phi[f] += (o_L - z_L) sum_k G_k (A_L,k - A_R,k)
//
// and hands up A_k = A_R,k + F_k (A_L,k - A_R,k), F_k the left edge's factor:
// z_L + z_R = 1 and o_L + o_R = 1, so the right edge's factor is 1 - F_k and
// its difference the left one's negative. A feature already split on above
// (its latest edge at level p, merged fraction z_p, factor f_p, d_p = o_p -
// z_p; o_p one bit per row) has the left factor replaced by rho = F / f_p and
// the difference by (d_L - d_p rho) / f_p, which takes its earlier edge's
// share back out; a row off at the earlier edge (o_p = 0) has rho the plain
// cover fraction and adds nothing. One pass per tree then costs a few
// operations per node and point where a path costs its length squared: at
// depth 8 about 32 FP64 operations for an inner node and 10 for a parent of
// two leaves, against 170 for each leaf's path.
//
// A lane is a row and a warp walks one tree at a time, all lanes alike, from
// shared memory: the nodes lie in preorder, and the walk is a nest of
// two-step loops, one per level, with every level's G and A in registers. A
// CTA's warps take different trees for the same 32 rows, each into its own
// FP64 slice; the CTAs of a cluster share a tile of rows where the tiles are
// few, and below 256 rows the trees are split through a workspace. Everything
// is summed in a fixed order. 1,000 trees of depth 8 over 28 features: 100,000
// rows in 55 ms (the path form: 249), 100 rows from the host in 183 us (810).
// At 20,000 rows it issues 53% of the time with 12 warps an SM (a G and an A
// of four doubles per level fill the registers), waiting on the chains of FP64
// operations; the FP64 pipe is 23% busy.

// warps a CTA has registers for (162, 116 and 76 a thread)
__host__ __device__ constexpr uint32_t tree_warps(uint32_t D)
{
    return D == 8 ? 12 : (D == 6 ? 16 : 24);
}
constexpr uint32_t k_tree_rows  = 32;
constexpr size_t   k_tree_smem  = 227 * 1024;
constexpr uint32_t k_tree_split = 256; // batches below this many rows split the trees

// A node's record. Leaf children hold their values here; the record of a
// feature split on above is followed by a MergedRec.
struct NodeRec
{
    uint32_t ff;   // feature | flags << 16
    uint32_t cond; // split bin | missing bin << 16
    float    vl, vr;
    double   zl;   // the left edge's merged cover fraction
    double   frac; // and its own
};
struct MergedRec
{
    double dp; // 1 - z_p
    double pad;
    double r[4]; // 1 / (z_p + (1 - z_p) t_k)
};
constexpr uint32_t k_nr_left   = 1u << 16; // the left child is a leaf
constexpr uint32_t k_nr_right  = 1u << 17;
constexpr uint32_t k_nr_dl     = 1u << 18; // missing goes left
constexpr uint32_t k_nr_merged = 1u << 19;
constexpr uint32_t k_nr_level  = 20; // the earlier edge's level, 4 bits

// Shared loads the compiler may neither merge nor keep across a subtree.
__device__ __forceinline__ uint4 lds_u4(uint32_t a)
{
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(a));
    return v;
}
__device__ __forceinline__ double2 lds_d2(uint32_t a)
{
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
    return v;
}

template <uint32_t M> struct TreeWalk
{
    uint16_t const *codes; // this lane's codes, a feature every k_tree_rows
    double         *phi;   // this lane's slice, likewise
    uint32_t        at;    // shared address of the next record
    uint32_t        on;    // bit L: the row is on at the path's level-L edge
    uint32_t        went;  // bit L: the row goes left at the path's level-L node
    double          t[M];
};

// The node at w.at, at level L of at most D: G its path's product, A what it
// hands up.
template <uint32_t D, uint32_t M, uint32_t L>
__device__ __forceinline__ void tree_node(TreeWalk<M> &w, double const (&G)[M], double (&A)[M])
{
    uint32_t const rec    = w.at;
    uint4 const    h      = lds_u4(rec);
    double2 const  z      = lds_d2(rec + 16);
    uint32_t const f      = (h.x & 0xFFFFu) * k_tree_rows;
    bool const     merged = L > 0 && (h.x & k_nr_merged) != 0;
    w.at                  = rec + sizeof(NodeRec) + (merged ? sizeof(MergedRec) : 0);
    uint32_t const code   = w.codes[f];
    bool const     left = code == (h.y >> 16) ? (h.x & k_nr_dl) != 0 : code <= (h.y & 0xFFFFu);
    bool const     onp  = !merged || ((w.on >> ((h.x >> k_nr_level) & 15u)) & 1u) != 0;
    double const   d    = (left && onp ? 1.0 : 0.0) - z.x;
    if (L + 1 == D || (h.x & (k_nr_left | k_nr_right)) == (k_nr_left | k_nr_right))
    {
        double const vr = __uint_as_float(h.w);
        double const q  = static_cast<double>(__uint_as_float(h.z)) - vr;
        double       add;
        if (!merged)
        {
            double const c1 = d * q;
            double const c0 = __fma_rn(z.x, q, vr);
            double       sg = G[0];
#pragma unroll
            for (uint32_t k = 1; k < M; ++k)
            {
                sg += G[k];
            }
#pragma unroll
            for (uint32_t k = 0; k < M; ++k)
            {
                A[k] = __fma_rn(w.t[k], c1, c0);
            }
            add = c1 * sg;
        }
        else
        {
            double const dp = lds_d2(rec + 32).x;
            double       sg = 0.0;
#pragma unroll
            for (uint32_t k = 0; k < M; k += 2)
            {
                double2 const r2 = lds_d2(rec + 48 + (k * 8));
#pragma unroll
                for (uint32_t kk = k; kk < k + 2 && kk < M; ++kk)
                {
                    double const r   = kk == k ? r2.x : r2.y;
                    double const rho = onp ? __fma_rn(d, w.t[kk], z.x) * r : z.y;
                    A[kk]            = __fma_rn(rho, q, vr);
                    sg               = __fma_rn(G[kk] * r, __fma_rn(-dp, rho, d), sg);
                }
            }
            add = onp ? q * sg : 0.0;
        }
        w.phi[f] += add;
        return;
    }
    if constexpr (L + 1 < D)
    {
        constexpr uint32_t below = (1u << L) - 1u;
        double             GX[M];
        double             AL[M];
#pragma unroll
        for (uint32_t k = 0; k < M; ++k)
        {
            GX[k] = __fma_rn(d, w.t[k], z.x);
        }
        if (merged)
        {
#pragma unroll
            for (uint32_t k = 0; k < M; k += 2)
            {
                double2 const r2 = lds_d2(rec + 48 + (k * 8));
                GX[k]            = onp ? GX[k] * r2.x : z.y;
                if (k + 1 < M)
                {
                    GX[k + 1] = onp ? GX[k + 1] * r2.y : z.y;
                }
            }
        }
#pragma unroll
        for (uint32_t k = 0; k < M; ++k)
        {
            GX[k] *= G[k];
        }
        w.went       = (w.went & below) | (left ? 1u << L : 0u);
        w.on         = (w.on & below) | (left && onp ? 1u << L : 0u);
        uint32_t leaf = h.x & k_nr_left;
        float    v    = __uint_as_float(h.z);
#pragma unroll 1
        for (uint32_t side = 0;; ++side)
        {
            if (leaf != 0)
            {
                double const vd = v;
#pragma unroll
                for (uint32_t k = 0; k < M; ++k)
                {
                    A[k] = vd;
                }
            }
            else
            {
                tree_node<D, M, L + 1>(w, GX, A);
            }
            if (side == 1)
            {
                break;
            }
            // over to the right child
            uint4 const    hh  = lds_u4(rec);
            uint32_t const lev = (hh.x >> k_nr_level) & 15u;
            bool const     po  = L == 0 || (hh.x & k_nr_merged) == 0 || ((w.on >> lev) & 1u) != 0;
            bool const     wr  = ((w.went >> L) & 1u) == 0;
            w.on               = (w.on & below) | (wr && po ? 1u << L : 0u);
            leaf               = hh.x & k_nr_right;
            v                  = __uint_as_float(hh.w);
#pragma unroll
            for (uint32_t k = 0; k < M; ++k)
            {
                AL[k] = A[k];
                GX[k] = G[k] - GX[k];
            }
        }
        uint4 const    hh = lds_u4(rec);
        double2 const  zz = lds_d2(rec + 16);
        uint32_t const ff = (hh.x & 0xFFFFu) * k_tree_rows;
        bool const     mm = L > 0 && (hh.x & k_nr_merged) != 0;
        bool const po = !mm || ((w.on >> ((hh.x >> k_nr_level) & 15u)) & 1u) != 0;
        bool const lo = ((w.went >> L) & 1u) != 0 && po;
        double const dd = (lo ? 1.0 : 0.0) - zz.x;
        double       sg = 0.0;
        if (!mm)
        {
#pragma unroll
            for (uint32_t k = 0; k < M; ++k)
            {
                double const q = AL[k] - A[k];
                A[k]           = __fma_rn(__fma_rn(dd, w.t[k], zz.x), q, A[k]);
                sg             = __fma_rn(G[k], q, sg);
            }
            sg *= dd;
        }
        else
        {
            double const dp = lds_d2(rec + 32).x;
#pragma unroll
            for (uint32_t k = 0; k < M; k += 2)
            {
                double2 const r2 = lds_d2(rec + 48 + (k * 8));
#pragma unroll
                for (uint32_t kk = k; kk < k + 2 && kk < M; ++kk)
                {
                    double const r   = kk == k ? r2.x : r2.y;
                    double const q   = AL[kk] - A[kk];
                    double const rho = po ? __fma_rn(dd, w.t[kk], zz.x) * r : zz.y;
                    A[kk]            = __fma_rn(rho, q, A[kk]);
                    sg = __fma_rn(G[kk] * q, __fma_rn(-dp, rho, dd) * r, sg);
                }
            }
            sg = po ? sg : 0.0;
        }
        w.phi[ff] += sg;
    }
}

// Small batches of deep trees give a warp a subtree: a tree is one warp's chain of
// dependent operations (depth 8: 80 us), and a few rows leave most warps idle. A
// node's sum is linear in A_L and A_R, so a subtree's warp adds its own part of
// every node above it: with A_s what the subtree hands up times the edges' factors
// from a node's child down to it, plus or minus sum_k G_k (...) A_s,k there. The
// units are the subtrees at level J (3, or 2 up to depth 6), and leaves above it. (28 features,
// depth 8, one row: 100 trees 96 us a warp per tree, 33 so; 1,000 trees 94 and
// 80; a path at a time, as deeper ensembles take it, 50 and 70.)
struct TreeUnit
{
    uint32_t rec[3];     // the records above it, offsets in the blob
    uint32_t begin, end; // its own; none: a leaf
    float    leaf;
    uint32_t len;        // records above it
    uint32_t dirs;       // bit l: left at the path's level l
};
constexpr uint32_t k_unit_levels = 3;
constexpr uint32_t k_unit_rec    = sizeof(NodeRec) + sizeof(MergedRec);
constexpr uint32_t k_unit_path   = k_unit_levels * k_unit_rec; // bytes before a subtree's records

// Levels above the units of a plan of at most D levels.
__host__ __device__ constexpr uint32_t unit_levels(uint32_t D)
{
    return D == 8 ? 3 : (D == 6 ? 2 : 0);
}

// The unit u below its path's level-L node (at level L = u.len: the unit itself),
// its records at shared address `first`.
template <uint32_t D, uint32_t M, uint32_t J, uint32_t L>
__device__ __forceinline__ void unit_node(TreeWalk<M> &w, TreeUnit const &u, uint32_t first,
                                          double const (&G)[M], double (&A)[M])
{
    if constexpr (L == J)
    {
        if (u.begin != u.end)
        {
            w.at = first + k_unit_path;
            tree_node<D, M, L>(w, G, A);
            return;
        }
    }
    if (u.len == L)
    {
        double const vd = u.leaf;
#pragma unroll
        for (uint32_t k = 0; k < M; ++k)
        {
            A[k] = vd;
        }
        return;
    }
    if constexpr (L < J)
    {
        uint32_t const rec    = first + (L * k_unit_rec);
        uint4 const    h      = lds_u4(rec);
        double2 const  z      = lds_d2(rec + 16);
        uint32_t const f      = (h.x & 0xFFFFu) * k_tree_rows;
        bool const     merged = L > 0 && (h.x & k_nr_merged) != 0;
        uint32_t const code   = w.codes[f];
        bool const     left = code == (h.y >> 16) ? (h.x & k_nr_dl) != 0 : code <= (h.y & 0xFFFFu);
        bool const     onp  = !merged || ((w.on >> ((h.x >> k_nr_level) & 15u)) & 1u) != 0;
        double const   d    = (left && onp ? 1.0 : 0.0) - z.x;
        double const   dp   = merged ? lds_d2(rec + 32).x : 0.0;
        bool const     down = ((u.dirs >> L) & 1u) != 0; // to the left
        w.on |= (down == left) && onp ? 1u << L : 0u;
        // (the earlier edge's 1 / f_p: 1 where there is none)
        auto const r = [&](uint32_t k)
        {
            if (!merged)
            {
                return 1.0;
            }
            double2 const r2 = lds_d2(rec + 48 + ((k & ~1u) * 8));
            return (k & 1u) == 0 ? r2.x : r2.y;
        };
        auto const rho = [&](uint32_t k) { return onp ? __fma_rn(d, w.t[k], z.x) * r(k) : z.y; };
        double     GX[M];
#pragma unroll
        for (uint32_t k = 0; k < M; ++k)
        {
            double const x = rho(k) * G[k];
            GX[k]          = down ? x : G[k] - x;
        }
        unit_node<D, M, J, L + 1>(w, u, first, GX, A);
        double sg = 0.0;
#pragma unroll
        for (uint32_t k = 0; k < M; ++k)
        {
            double const x = rho(k);
            sg             = __fma_rn(G[k] * A[k], __fma_rn(-dp, x, d) * r(k), sg);
            A[k] *= down ? x : 1.0 - x;
        }
        w.phi[f] += onp ? (down ? sg : -sg) : 0.0;
    }
}

__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_size()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
// A double of another CTA of the cluster, at this CTA's shared address a.
__device__ __forceinline__ double ld_cluster(uint32_t a, uint32_t rank)
{
    uint32_t r;
    double   v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(r));
    return v;
}

// grid (cluster CTAs x row tiles, splits), blockDim.x / 32 warps: warp v of
// the cluster and split takes trees v, v + V, v + 2 V ... of all V warps that
// share its rows (J > 0: units). A split writes its raw sums into ws, the only
// split composes the row.
template <uint32_t D, uint32_t J>
__global__ void __launch_bounds__(tree_warps(D) * 32, 1)
    shap_tree_kernel(uint8_t const *__restrict__ bins8, uint16_t const *__restrict__ bins16,
                     uint64_t n_pad, uint64_t n_rows, uint32_t F,
                     unsigned char const *__restrict__ blob, uint32_t const *__restrict__ blob_off,
                     TreeUnit const *__restrict__ units, uint32_t n_trees, uint32_t room, Gauss g, double lr, double bias, double init,
                     double *__restrict__ out, double *__restrict__ ws)
{
    constexpr uint32_t M = D / 2;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t const T     = blockDim.x;
    uint32_t const W     = T / 32;
    uint32_t const lane  = threadIdx.x & 31;
    uint32_t const wid   = threadIdx.x >> 5;
    uint32_t const C     = cluster_size();
    uint32_t const rank  = cluster_rank();
    uint32_t const slice = (F + 1) * k_tree_rows;
    auto *const    phi_s = reinterpret_cast<double *>(smem); // [warp][F + 1][rows]
    unsigned char *tree_s = smem + (size_t{W} * slice * 8);  // [warp][room]
    auto *const codes_s   = reinterpret_cast<uint16_t *>(tree_s + (size_t{W} * room)); // [F][rows]
    uint64_t const row0   = static_cast<uint64_t>(blockIdx.x / C) * k_tree_rows;
    for (uint32_t i = threadIdx.x; i < F * k_tree_rows; i += T)
    {
        uint32_t const f = i / k_tree_rows;
        uint64_t const r = row0 + (i % k_tree_rows);
        uint32_t       c = 0;
        if (r < n_rows)
        {
            c = bins8 != nullptr ? bins8[(static_cast<uint64_t>(f) * n_pad) + r]
                                 : bins16[(static_cast<uint64_t>(f) * n_pad) + r];
        }
        codes_s[i] = static_cast<uint16_t>(c);
    }
    for (uint32_t i = threadIdx.x; i < W * slice; i += T)
    {
        phi_s[i] = 0.0;
    }
    __syncthreads();
    TreeWalk<M> w;
    w.codes = codes_s + lane;
    w.phi   = phi_s + (wid * slice) + lane;
    w.on    = 0;
    w.went  = 0;
    double G[M];
#pragma unroll
    for (uint32_t k = 0; k < M; ++k)
    {
        w.t[k] = g.x[k];
        G[k]   = g.w[k];
    }
    unsigned char *const mine  = tree_s + (size_t{wid} * room);
    uint32_t const       first = static_cast<uint32_t>(__cvta_generic_to_shared(mine));
    uint32_t const       V     = gridDim.y * C * W;
    for (uint32_t t = (((blockIdx.y * C) + rank) * W) + wid; t < n_trees; t += V)
    {
        if constexpr (J > 0)
        {
            TreeUnit const u = units[t];
            __syncwarp(); // the previous unit is done
#pragma unroll
            for (uint32_t l = 0; l < J; ++l)
            {
                // (a record alone may be shorter: what follows it is not read)
                if (l < u.len && lane < k_unit_rec / 16)
                {
                    *reinterpret_cast<uint4 *>(mine + (l * k_unit_rec) + (lane * 16)) =
                        __ldg(reinterpret_cast<uint4 const *>(blob + u.rec[l]) + lane);
                }
            }
            for (uint32_t x = lane * 16; x < u.end - u.begin; x += 512)
            {
                *reinterpret_cast<uint4 *>(mine + k_unit_path + x) =
                    __ldg(reinterpret_cast<uint4 const *>(blob + u.begin + x));
            }
            __syncwarp();
            double A[M];
            w.on   = 0;
            w.went = 0;
            unit_node<D, M, J, 0>(w, u, first, G, A);
            continue;
        }
        uint32_t const b0 = blob_off[t];
        uint32_t const nb = blob_off[t + 1] - b0;
        __syncwarp(); // the previous tree is done
        for (uint32_t x = lane * 16; x < nb; x += 512)
        {
            *reinterpret_cast<uint4 *>(mine + x) =
                __ldg(reinterpret_cast<uint4 const *>(blob + b0 + x));
        }
        __syncwarp();
        if (nb != 0) // (a tree of one leaf has no nodes)
        {
            double A[M];
            w.at = first;
            tree_node<D, M, 0>(w, G, A);
        }
    }
    __syncthreads();
    // the warps' slices, into the first one
    for (uint32_t i = threadIdx.x; i < slice; i += T)
    {
        double s = phi_s[i];
        for (uint32_t v = 1; v < W; ++v)
        {
            s += phi_s[(v * slice) + i];
        }
        phi_s[i] = s;
    }
    if (C > 1)
    {
        cluster_sync();
    }
    else
    {
        __syncthreads();
    }
    // the cluster's CTAs in order, each CTA a share of the tile's rows
    uint32_t const rows = k_tree_rows / C; // C is 1, 2, 4 or 8
    for (uint32_t i = threadIdx.x; i < rows * (F + 1); i += T)
    {
        uint32_t const rl = (rank * rows) + (i / (F + 1));
        uint32_t const f  = i % (F + 1);
        uint64_t const r  = row0 + rl;
        if (r >= n_rows)
        {
            continue;
        }
        double const *cell = phi_s + (f * k_tree_rows) + rl;
        double        s    = 0.0;
        if (C == 1)
        {
            s = *cell;
        }
        else
        {
            uint32_t const a = static_cast<uint32_t>(__cvta_generic_to_shared(cell));
            for (uint32_t q = 0; q < C; ++q)
            {
                s += ld_cluster(a, q);
            }
        }
        if (ws == nullptr)
        {
            out[(r * (F + 1)) + f] = f == F ? ((s + bias) * lr) + init : s * lr;
        }
        else
        {
            ws[((static_cast<uint64_t>(blockIdx.y) * n_rows + r) * (F + 1)) + f] = s;
        }
    }
    if (C > 1)
    {
        cluster_sync(); // no CTA leaves while another reads its slice
    }
}

// The tree splits' sums, composed: a warp per cell, its lanes every 32nd split.
__global__ void __launch_bounds__(256)
    shap_tree_reduce_kernel(double const *__restrict__ ws, uint64_t n, uint32_t F,
                            uint32_t splits, double lr, double bias, double init,
                            double *__restrict__ out)
{
    uint64_t const i    = (static_cast<uint64_t>(blockIdx.x) * 8) + (threadIdx.x >> 5);
    uint32_t const lane = threadIdx.x & 31;
    if (i >= n)
    {
        return;
    }
    double s = 0.0;
    for (uint32_t k = lane; k < splits; k += 32)
    {
        s += ws[(static_cast<uint64_t>(k) * n) + i];
    }
#pragma unroll
    for (uint32_t o = 16; o > 0; o >>= 1)
    {
        s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    }
    if (lane == 0)
    {
        out[i] = i % (F + 1) == F ? ((s + bias) * lr) + init : s * lr;
    }
}

// Gauss-Legendre nodes and weights on [0, 1]: the roots of the degree-m
// Legendre polynomial by Newton's method on the three-term recurrence,
// weights 2 / ((1 - x^2) P'(x)^2), mapped from [-1, 1].
void gauss_legendre(uint32_t m, std::vector<double> &x01, std::vector<double> &w01)
{
    x01.assign(m, 0.0);
    w01.assign(m, 0.0);
    double const pi = 3.14159265358979323846;
    for (uint32_t i = 0; i < m; ++i)
    {
        double x = std::cos(pi * (i + 0.75) / (m + 0.5));
        double dp = 0.0;
        for (int it = 0; it < 100; ++it)
        {
            double p0 = 1.0;
            double p1 = x;
            for (uint32_t k = 2; k <= m; ++k)
            {
                double const p2 = (((2.0 * k) - 1.0) * x * p1 - ((k - 1.0) * p0)) / k;
                p0              = p1;
                p1              = p2;
            }
            double const pm = m == 0 ? 1.0 : (m == 1 ? x : p1);
            double const pmm1 = m == 1 ? 1.0 : p0;
            dp                = m * (x * pm - pmm1) / ((x * x) - 1.0);
            double const dx   = pm / dp;
            x -= dx;
            if (std::fabs(dx) < 1e-16)
            {
                break;
            }
        }
        x01[i] = 0.5 * (x + 1.0);
        w01[i] = 1.0 / ((1.0 - (x * x)) * dp * dp); // 2 / (...) on [-1,1], halved
    }
}

struct Packed
{
    std::vector<PathHead> paths;
    std::vector<uint32_t> first; // each path's first element in elems
    std::vector<PathElem> elems;
    uint32_t              max_len = 0;
};

struct TreeView
{
    uint32_t const *feature;
    uint32_t const *split_bin;
    uint32_t const *left;
    uint32_t const *right;
    uint8_t const  *dl;
    float const    *value;
    float const    *cover;
    uint32_t        n;
};

// tree_expected_value (src/shap.cpp:250-290): cover-weighted leaf mean.
double expected_value(TreeView const &t, uint32_t id)
{
    if (t.feature[id] == k_leaf_flag)
    {
        return t.value[id];
    }
    double const cover = t.cover[id];
    if (cover <= 0.0)
    {
        return 0.0;
    }
    return ((static_cast<double>(t.cover[t.left[id]]) * expected_value(t, t.left[id])) +
            (static_cast<double>(t.cover[t.right[id]]) * expected_value(t, t.right[id]))) /
           cover;
}

struct Cond
{
    uint32_t feature;
    uint32_t lo, hi; // passing non-missing bins [lo, hi]
    bool     miss_ok;
    double   zero;
};

// Every root-to-leaf path of one tree, conditions on one feature merged:
// left at split s keeps bins <= s (and missing when default_left), right
// keeps bins > s (and missing otherwise), cover fractions multiply.
void collect(TreeView const &t, uint32_t const *last, uint32_t id, std::vector<Cond> &path,
             Packed &out)
{
    if (t.feature[id] == k_leaf_flag)
    {
        PathHead const h{static_cast<double>(t.value[id]), static_cast<uint32_t>(path.size()),
                         0u};
        out.first.push_back(static_cast<uint32_t>(out.elems.size()));
        for (Cond const &c : path)
        {
            out.elems.push_back({c.feature | (c.miss_ok ? 0x80000000u : 0u),
                                 (c.lo & 0xFFFFu) | ((c.hi & 0xFFFFu) << 16), c.zero});
        }
        out.max_len = std::max<uint32_t>(out.max_len, h.count);
        out.paths.push_back(h);
        return;
    }
    uint32_t const f     = t.feature[id];
    double const   cover = t.cover[id];
    for (int side = 0; side < 2; ++side)
    {
        uint32_t const child = side == 0 ? t.left[id] : t.right[id];
        double const   frac  = cover > 0.0 ? static_cast<double>(t.cover[child]) / cover : 0.0;
        size_t         k     = 0;
        while (k < path.size() && path[k].feature != f)
        {
            ++k;
        }
        bool const fresh = k == path.size();
        Cond const saved = fresh ? Cond{} : path[k];
        if (fresh)
        {
            path.push_back({f, 0, last[f] - 1, true, 1.0});
        }
        Cond &c = path[k];
        if (side == 0)
        {
            c.hi      = std::min(c.hi, t.split_bin[id]);
            c.miss_ok = c.miss_ok && t.dl[id] != 0;
        }
        else
        {
            c.lo      = std::max(c.lo, t.split_bin[id] + 1);
            c.miss_ok = c.miss_ok && t.dl[id] == 0;
        }
        c.zero *= frac;
        collect(t, last, child, path, out);
        if (fresh)
        {
            path.pop_back();
        }
        else
        {
            path[k] = saved;
        }
    }
}

// The tree form's blob: each tree's records in preorder.
struct TreeBlob
{
    std::vector<unsigned char> bytes;
    std::vector<uint32_t>      off; // n_trees + 1
    uint32_t                   room = 0;
    // the units at level J (0: none): a path's records so far, and theirs
    uint32_t              J         = 0;
    uint32_t              unit_room = 0;
    uint64_t              nodes     = 0;
    uint32_t              rec[k_unit_levels] = {};
    std::vector<TreeUnit> units;
};

// Levels of split nodes; 0 where the tree form cannot take the tree (over 8
// levels, or covers that do not add up).
uint32_t tree_levels(TreeView const &t, uint32_t id, uint32_t level)
{
    if (level == 8)
    {
        return 0;
    }
    double const c = t.cover[id];
    if (!(c > 0.0) || static_cast<double>(t.cover[t.left[id]]) + t.cover[t.right[id]] != c)
    {
        return 0;
    }
    uint32_t most = 1;
    for (uint32_t const child : {t.left[id], t.right[id]})
    {
        if (t.feature[child] != k_leaf_flag)
        {
            uint32_t const m = tree_levels(t, child, level + 1);
            if (m == 0)
            {
                return 0;
            }
            most = std::max(most, m + 1);
        }
    }
    return most;
}

struct PathEdge
{
    uint32_t feature;
    double   z; // merged cover fraction
};

// Node id's subtree; dirs: the path's left turns, bit by level.
void pack_node(TreeView const &t, uint32_t const *last, uint32_t id, std::vector<PathEdge> &path,
               std::vector<double> const &gx, TreeBlob &tb, uint32_t dirs)
{
    std::vector<unsigned char> &out   = tb.bytes;
    uint32_t const              level = static_cast<uint32_t>(path.size());
    uint32_t const              begin = static_cast<uint32_t>(out.size());
    auto const                  unit  = [&](uint32_t b, uint32_t e, float leaf, uint32_t len, uint32_t d)
    {
        tb.units.push_back({{tb.rec[0], tb.rec[1], tb.rec[2]}, b, e, leaf, len, d});
        tb.unit_room = std::max(tb.unit_room, k_unit_path + (e - b));
    };
    ++tb.nodes;
    if (level < tb.J)
    {
        tb.rec[level] = begin;
    }
    uint32_t const f     = t.feature[id];
    uint32_t const l     = t.left[id];
    uint32_t const r     = t.right[id];
    double const   cover = t.cover[id];
    double const   fl    = static_cast<double>(t.cover[l]) / cover;
    double const   fr    = static_cast<double>(t.cover[r]) / cover;
    uint32_t       prev  = static_cast<uint32_t>(path.size());
    while (prev > 0 && path[prev - 1].feature != f)
    {
        --prev;
    }
    bool const   merged = prev > 0;
    double const zp     = merged ? path[prev - 1].z : 1.0;
    NodeRec      n{};
    n.ff   = f | (t.feature[l] == k_leaf_flag ? k_nr_left : 0u) |
           (t.feature[r] == k_leaf_flag ? k_nr_right : 0u) | (t.dl[id] != 0 ? k_nr_dl : 0u) |
           (merged ? k_nr_merged | ((prev - 1) << k_nr_level) : 0u);
    n.cond = t.split_bin[id] | (last[f] << 16);
    n.vl   = t.value[l];
    n.vr   = t.value[r];
    n.zl   = zp * fl;
    n.frac = fl;
    auto const *nb = reinterpret_cast<unsigned char const *>(&n);
    out.insert(out.end(), nb, nb + sizeof(n));
    if (merged)
    {
        MergedRec m{};
        m.dp = 1.0 - zp;
        for (size_t k = 0; k < gx.size(); ++k)
        {
            m.r[k] = 1.0 / (zp + ((1.0 - zp) * gx[k]));
        }
        auto const *mb = reinterpret_cast<unsigned char const *>(&m);
        out.insert(out.end(), mb, mb + sizeof(m));
    }
    for (int side = 0; side < 2; ++side)
    {
        uint32_t const child = side == 0 ? l : r;
        uint32_t const d     = dirs | (side == 0 ? 1u << level : 0u);
        if (t.feature[child] != k_leaf_flag)
        {
            path.push_back({f, zp * (side == 0 ? fl : fr)});
            pack_node(t, last, child, path, gx, tb, d);
            path.pop_back();
        }
        else if (level < tb.J)
        {
            unit(0, 0, t.value[child], level + 1, d);
        }
    }
    if (level == tb.J && tb.J > 0)
    {
        unit(begin, static_cast<uint32_t>(out.size()), 0.0F, level, dirs);
    }
}

} // namespace

// A device buffer released with its owner.
struct ShapBuf
{
    void *p = nullptr;
    ShapBuf() = default;
    ShapBuf(ShapBuf const &) = delete;
    ShapBuf &operator=(ShapBuf const &) = delete;
    ~ShapBuf()
    {
        if (p != nullptr)
        {
            cudaFree(p);
        }
    }
    void alloc(size_t bytes)
    {
        check(cudaMalloc(&p, std::max<size_t>(bytes, 16)), "cudaMalloc");
    }
    void upload(void const *src, size_t bytes)
    {
        alloc(bytes);
        if (bytes > 0)
        {
            check(cudaMemcpy(p, src, bytes, cudaMemcpyHostToDevice), "cudaMemcpy");
        }
    }
    void grow(size_t bytes, size_t &cap)
    {
        if (cap >= bytes)
        {
            return;
        }
        if (p != nullptr)
        {
            check(cudaFree(p), "cudaFree");
            p   = nullptr;
            cap = 0;
        }
        check(cudaMalloc(&p, bytes), "cudaMalloc");
        cap = bytes;
    }
    template <typename T> T *as() const
    {
        return static_cast<T *>(p);
    }
};

} // namespace bb

struct bb_shap_plan
{
    uint32_t              n_feats = 0;
    bool                  u8      = true;
    std::vector<uint32_t> cut_off;
    uint32_t              K       = 8;
    uint32_t              n_paths = 0;
    double                bias    = 0.0;
    double                lr      = 0.0;
    double                init    = 0.0;
    bb::Gauss             gauss{};
    bb::ShapBuf           heads, elems, last;
    // the tree form (tree_depth > 0): its blob, warps per CTA, and the
    // resident CTAs of the GPU by cluster size 1, 2, 4, 8
    uint32_t              tree_depth = 0;
    uint32_t              n_trees    = 0;
    uint32_t              room       = 0;
    uint32_t              warps      = 0;
    uint32_t              resident[4] = {};
    uint32_t              unit_level = 0; // small batches' units: their level (0: none)
    uint32_t              n_units    = 0;
    uint32_t              unit_room  = 0;
    uint32_t              unit_warps = 0;
    double                tree_cost = 0.0; // nodes of a tree, and of a unit with its path
    double                unit_cost = 0.0;
    bb::ShapBuf           tables; // of the tree form: the three below
    uint32_t             *blob_off = nullptr;
    bb::TreeUnit         *units    = nullptr;
    unsigned char        *blob     = nullptr;
    std::mutex            mu;
    bb::ShapBuf           ws, out;
    size_t                ws_cap = 0, out_cap = 0;
    cudaStream_t          stream = nullptr;
    ~bb_shap_plan()
    {
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

using TreeFn = void (*)(uint8_t const *, uint16_t const *, uint64_t, uint64_t, uint32_t,
                        unsigned char const *, uint32_t const *, TreeUnit const *, uint32_t,
                        uint32_t, Gauss, double, double, double, double *, double *);

// J: the units' level, 0 for whole trees.
TreeFn tree_fn(uint32_t D, uint32_t J)
{
    switch ((10 * D) + J)
    {
    case 40: return shap_tree_kernel<4, 0>;
    case 60: return shap_tree_kernel<6, 0>;
    case 62: return shap_tree_kernel<6, 2>;
    case 80: return shap_tree_kernel<8, 0>;
    case 83: return shap_tree_kernel<8, 3>;
    default: throw std::logic_error("bb_shap_plan: no such tree form");
    }
}

size_t tree_smem(uint32_t F, uint32_t room, uint32_t warps)
{
    return (size_t{warps} * (((size_t{F} + 1) * k_tree_rows * sizeof(double)) + room)) +
           (size_t{F} * k_tree_rows * sizeof(uint16_t));
}

cudaLaunchConfig_t tree_config(cudaLaunchAttribute *at, uint32_t cluster, dim3 grid,
                               uint32_t warps, size_t smem, cudaStream_t s)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim          = grid;
    cfg.blockDim         = dim3(warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream           = s;
    at->id               = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim   = {cluster, 1, 1};
    cfg.attrs            = at;
    cfg.numAttrs         = 1;
    return cfg;
}

// The tree form of an ensemble of `depth` levels, or null where two warps'
// slices and trees do not fit a CTA's shared memory.
std::unique_ptr<bb_shap_plan> make_tree_plan(std::vector<TreeView> const &views,
                                             std::vector<uint32_t> const &last, uint32_t depth)
{
    auto           pl = std::make_unique<bb_shap_plan>();
    uint32_t const F  = static_cast<uint32_t>(last.size());
    uint32_t const D  = depth <= 4 ? 4 : (depth <= 6 ? 6 : 8);
    uint32_t const m  = D / 2; // exact for up to D elements on a path
    std::vector<double> gx;
    std::vector<double> gw;
    gauss_legendre(m, gx, gw);
    pl->gauss.m = m;
    for (uint32_t k = 0; k < m; ++k)
    {
        pl->gauss.x[k] = gx[k];
        pl->gauss.w[k] = gw[k];
    }
    TreeBlob              tb;
    std::vector<PathEdge> path;
    // (trees for several rounds of all the GPU's warps even them out by themselves)
    tb.J = views.size() < size_t{4} * k_sms * tree_warps(D) ? unit_levels(D) : 0;
    for (TreeView const &tv : views)
    {
        tb.off.push_back(static_cast<uint32_t>(tb.bytes.size()));
        if (tv.feature[0] != k_leaf_flag)
        {
            pack_node(tv, last.data(), 0, path, gx, tb, 0);
        }
        if (tb.bytes.size() > 0x7FFFFFFFu)
        {
            return nullptr; // 32-bit offsets
        }
        tb.room = std::max(tb.room, static_cast<uint32_t>(tb.bytes.size()) - tb.off.back());
    }
    tb.off.push_back(static_cast<uint32_t>(tb.bytes.size()));
    // the warps whose slices and trees (or units) of `room` bytes fit a CTA
    auto const warps = [&](uint32_t room)
    {
        size_t const one = tree_smem(F, room, 1) - tree_smem(F, room, 0);
        return static_cast<uint32_t>(
            std::min<size_t>(tree_warps(D), (k_tree_smem - tree_smem(F, room, 0)) / one));
    };
    pl->warps = warps(tb.room);
    if (pl->warps < 2)
    {
        return nullptr;
    }
    pl->tree_depth  = D;
    pl->n_trees     = static_cast<uint32_t>(views.size());
    pl->room        = tb.room;
    size_t const sm = tree_smem(F, tb.room, pl->warps);
    allow_smem(tree_fn(D, 0));
    for (uint32_t c = 0; c < 4; ++c)
    {
        cudaLaunchAttribute at{};
        cudaLaunchConfig_t  cfg = tree_config(&at, 1u << c, dim3(1u << c), pl->warps, sm, nullptr);
        int                 n   = 0;
        check(cudaOccupancyMaxActiveClusters(&n, tree_fn(D, 0), &cfg),
              "cudaOccupancyMaxActiveClusters");
        pl->resident[c] = static_cast<uint32_t>(n) << c;
    }
    if (tb.J > 0)
    {
        allow_smem(tree_fn(D, tb.J));
        pl->unit_level = tb.J;
        pl->n_units    = static_cast<uint32_t>(tb.units.size());
        pl->unit_room  = tb.unit_room;
        pl->unit_warps = std::max(1u, warps(pl->unit_room));
        pl->tree_cost  = static_cast<double>(tb.nodes) / static_cast<double>(views.size());
        pl->unit_cost  = (static_cast<double>(tb.nodes) / pl->n_units) + 8.0;
    }
    // the offsets, the units and the blob, in one allocation (a unit's path reads whole
    // records: some bytes past the blob, whatever they hold)
    auto const   lines = [](size_t n) { return (n + 127) & ~size_t{127}; };
    size_t const n_off = lines(tb.off.size() * 4);
    size_t const n_un  = lines(tb.units.size() * sizeof(TreeUnit));
    pl->tables.alloc(n_off + n_un + tb.bytes.size() + k_unit_rec);
    auto *const at = pl->tables.as<unsigned char>();
    pl->blob_off   = reinterpret_cast<uint32_t *>(at);
    pl->units      = reinterpret_cast<TreeUnit *>(at + n_off);
    pl->blob       = at + n_off + n_un;
    auto const up  = [](void *to, void const *from, size_t n)
    { check(cudaMemcpy(to, from, n, cudaMemcpyHostToDevice), "cudaMemcpy"); };
    up(pl->blob_off, tb.off.data(), tb.off.size() * 4);
    up(pl->units, tb.units.data(), tb.units.size() * sizeof(TreeUnit));
    up(pl->blob, tb.bytes.data(), tb.bytes.size());
    return pl;
}

std::unique_ptr<bb_shap_plan> make_shap_plan(Plane const &p, uint32_t n_trees,
                                             uint32_t const *roots, uint32_t n_nodes,
                                             uint32_t const *feature, uint32_t const *split_bin,
                                             uint32_t const *left, uint32_t const *right,
                                             uint8_t const *default_left, float const *value,
                                             float const *cover, float lr, float init)
{
    if (roots == nullptr || feature == nullptr || split_bin == nullptr || left == nullptr ||
        right == nullptr || default_left == nullptr || value == nullptr || cover == nullptr ||
        n_trees == 0)
    {
        throw std::invalid_argument("bb_shap_plan_create: null argument or empty ensemble");
    }
    uint32_t const F = p.n_feats;
    if (F > k_max_shap_feats)
    {
        throw ConfigError("bb_shap_plan_create: more than 128 features; use the host "
                          "TreeSHAP walk");
    }
    std::vector<uint32_t> last(F);
    for (uint32_t f = 0; f < F; ++f)
    {
        last[f] = p.h_cut_off[f + 1] - p.h_cut_off[f] - 1;
    }
    double                bias  = 0.0; // sum over trees of the expected values
    uint32_t              depth = 0;   // the tree form's levels
    bool                  trees = true;
    std::vector<TreeView> views;
    views.reserve(n_trees);
    for (uint32_t t = 0; t < n_trees; ++t)
    {
        uint32_t const b = roots[t];
        uint32_t const e = t + 1 < n_trees ? roots[t + 1] : n_nodes;
        if (!(b < e && e <= n_nodes))
        {
            throw std::invalid_argument("bb_shap_plan_create: bad tree roots");
        }
        for (uint32_t i = b; i < e; ++i)
        {
            if (feature[i] == k_leaf_flag)
            {
                continue;
            }
            if (feature[i] >= F || !(left[i] > i - b && right[i] > i - b &&
                                     b + left[i] < e && b + right[i] < e) ||
                split_bin[i] + 1 > last[feature[i]])
            {
                throw std::invalid_argument("bb_shap_plan_create: malformed tree");
            }
        }
        TreeView const tv{feature + b, split_bin + b, left + b, right + b,
                          default_left + b, value + b, cover + b, e - b};
        bias += expected_value(tv, 0);
        if (trees && tv.feature[0] != k_leaf_flag)
        {
            uint32_t const m = tree_levels(tv, 0, 0);
            trees            = m != 0;
            depth            = std::max(depth, m);
        }
        views.push_back(tv);
    }
    if (trees && depth > 0)
    {
        auto pl = make_tree_plan(views, last, depth);
        if (pl != nullptr)
        {
            pl->n_feats = F;
            pl->u8      = p.u8;
            pl->cut_off.assign(p.h_cut_off, p.h_cut_off + F + 1);
            pl->bias = bias;
            pl->lr   = static_cast<double>(lr);
            pl->init = static_cast<double>(init);
            check(cudaStreamCreateWithFlags(&pl->stream, cudaStreamNonBlocking),
                  "cudaStreamCreate");
            return pl;
        }
    }
    Packed pk;
    for (TreeView const &tv : views)
    {
        std::vector<Cond> path;
        collect(tv, last.data(), 0, path, pk);
    }
    if (pk.max_len > k_max_path)
    {
        throw ConfigError("bb_shap_plan_create: a path holds more than 32 distinct features");
    }
    auto pl     = std::make_unique<bb_shap_plan>();
    pl->n_feats = F;
    pl->u8      = p.u8;
    pl->cut_off.assign(p.h_cut_off, p.h_cut_off + F + 1);
    pl->K       = pk.max_len <= 8 ? 8u : (pk.max_len <= 16 ? 16u : 32u);
    pl->n_paths = static_cast<uint32_t>(pk.paths.size());
    pl->bias    = bias;
    pl->lr      = static_cast<double>(lr);
    pl->init    = static_cast<double>(init);
    uint32_t const      m = std::max<uint32_t>(1, (pk.max_len + 1) / 2);
    std::vector<double> gx;
    std::vector<double> gw;
    gauss_legendre(m, gx, gw);
    pl->gauss.m = m;
    for (uint32_t k = 0; k < m; ++k)
    {
        pl->gauss.x[k] = gx[k];
        pl->gauss.w[k] = gw[k];
    }
    // fixed-stride element records: path j's elements at [j * K, j * K + count)
    std::vector<PathElem> el(static_cast<size_t>(pl->n_paths) * pl->K, PathElem{0, 0, 1.0});
    for (uint32_t j = 0; j < pl->n_paths; ++j)
    {
        std::copy_n(pk.elems.begin() + pk.first[j], pk.paths[j].count,
                    el.begin() + (static_cast<size_t>(j) * pl->K));
    }
    pl->heads.upload(pk.paths.data(), pk.paths.size() * sizeof(PathHead));
    pl->elems.upload(el.data(), el.size() * sizeof(PathElem));
    pl->last.upload(last.data(), F * 4ull);
    check(cudaStreamCreateWithFlags(&pl->stream, cudaStreamNonBlocking), "cudaStreamCreate");
    return pl;
}

void shap_check_plane(bb_shap_plan const &pl, Plane const &p)
{
    if (p.n_feats != pl.n_feats || p.u8 != pl.u8 ||
        !std::equal(pl.cut_off.begin(), pl.cut_off.end(), p.h_cut_off))
    {
        throw std::invalid_argument(
            "bb_shap_plan: the plane's features or bin counts differ from the plan's");
    }
    if (p.n_rows > 0x7FFFFFFFull)
    {
        throw ConfigError("bb_shap_plan: more than 2^31 - 1 rows in one call");
    }
}

using TileFn = void (*)(uint8_t const *, uint16_t const *, uint64_t, uint64_t, uint32_t const *,
                        uint32_t, PathHead const *, PathElem const *, uint32_t, uint32_t,
                        uint32_t, uint32_t, Gauss, double, double, double, double *, double *);

TileFn tile_fn(uint32_t K)
{
    return K == 8 ? shap_tile_kernel<8> : (K == 16 ? shap_tile_kernel<16> : shap_tile_kernel<32>);
}

// The tree form's launch.
uint32_t tree_launch(bb_shap_plan &pl, Plane const &p, double *out, cudaStream_t s)
{
    uint64_t const n      = p.n_rows;
    uint32_t const F      = pl.n_feats;
    uint32_t const tiles  = ceil_div(n, k_tree_rows);
    uint32_t       J      = 0;
    uint32_t       count  = pl.n_trees;
    uint32_t       room   = pl.room;
    uint32_t       most   = pl.warps;
    uint32_t       W      = std::min(most, count);
    uint32_t       C      = 1;
    uint32_t       splits = 1;
    if (n < k_tree_split)
    {
        // about one CTA per SM, a tree (a unit) at a time in each of its warps: the
        // form whose rounds over them visit fewer nodes one after another (a unit's
        // path and its start are worth about eight)
        uint32_t const ctas  = std::max(1u, k_sms / tiles);
        double const   trees = pl.tree_cost * ceil_div(count, ctas * most);
        if (pl.unit_level > 0 &&
            pl.unit_cost * ceil_div(pl.n_units, ctas * pl.unit_warps) < trees)
        {
            J     = pl.unit_level;
            count = pl.n_units;
            room  = pl.unit_room;
            most  = pl.unit_warps;
        }
        splits = std::min(ctas, count);
        W      = std::min(most, ceil_div(count, splits));
        splits = std::min(splits, ceil_div(count, W));
        if (pl.tree_depth == 4 && count <= 8 * most && pl.resident[3] != 0)
        {
            // short trees: a cluster's warps take one each, without the second
            // launch that sums the splits
            C      = 8;
            W      = ceil_div(count, 8);
            splits = 1;
        }
    }
    else
    {
        // the cluster size whose waves of trees are the fewest: more CTAs per
        // tile fill a GPU that the tiles alone would not, or even out the
        // last wave (no workspace: launches on several streams may overlap)
        uint64_t best = ~uint64_t{0};
        for (uint32_t c = 0; c < 4; ++c)
        {
            if (pl.resident[c] == 0)
            {
                continue;
            }
            uint64_t const cost = static_cast<uint64_t>(ceil_div(uint64_t{tiles} << c,
                                                                 pl.resident[c])) *
                                  ceil_div(pl.n_trees, W << c);
            if (cost < best)
            {
                best = cost;
                C    = 1u << c;
            }
        }
    }
    double *ws = nullptr;
    if (splits > 1)
    {
        pl.ws.grow(static_cast<size_t>(splits) * n * (F + 1) * sizeof(double), pl.ws_cap);
        ws = pl.ws.as<double>();
    }
    cudaLaunchAttribute at{};
    cudaLaunchConfig_t  cfg = tree_config(&at, C, dim3(tiles * C, splits), W,
                                          tree_smem(F, room, W), s);
    check(cudaLaunchKernelEx(
              &cfg, tree_fn(pl.tree_depth, J),
              p.u8 ? static_cast<uint8_t const *>(p.bins) : static_cast<uint8_t const *>(nullptr),
              p.u8 ? static_cast<uint16_t const *>(nullptr) : static_cast<uint16_t const *>(p.bins),
              p.n_pad, n, F, static_cast<unsigned char const *>(pl.blob),
              static_cast<uint32_t const *>(pl.blob_off), static_cast<TreeUnit const *>(pl.units),
              count, room, pl.gauss, pl.lr,
              pl.bias, pl.init, out, ws),
          "shap_tree_kernel");
    if (splits == 1)
    {
        return 1;
    }
    uint64_t const cells = n * (F + 1);
    shap_tree_reduce_kernel<<<ceil_div(cells, 8), 256, 0, s>>>(ws, cells, F, splits, pl.lr,
                                                               pl.bias, pl.init, out);
    check(cudaGetLastError(), "shap_tree_reduce_kernel");
    return 2;
}

// Enqueues the contributions of every row of p into out (device,
// n_rows x (F + 1)); returns the kernels launched.
uint32_t shap_launch(bb_shap_plan &pl, Plane const &p, double *out, cudaStream_t s)
{
    uint64_t const n  = p.n_rows;
    if (n == 0)
    {
        return 0; // an empty request plane: nothing to explain
    }
    uint32_t const F  = pl.n_feats;
    if (pl.tree_depth > 0)
    {
        return tree_launch(pl, p, out, s);
    }
    TileFn const   fn = tile_fn(pl.K);
    // 128 threads while their FP64 slices fit 100 KB, else 64
    uint32_t const T   = (static_cast<size_t>(F) + 1) * 128 * 8 <= 102400 ? 128u : 64u;
    size_t const   rec = sizeof(PathHead) + ((pl.K + 1ull) * sizeof(PathElem));
    auto const chunk_of = [&](uint32_t PL)
    { return PL * std::max<uint32_t>(1, static_cast<uint32_t>(k_chunk_budget / (rec * PL))); };
    auto const smem_of = [&](uint32_t PL)
    {
        return ((static_cast<size_t>(F) + 1) * T * sizeof(double)) + (chunk_of(PL) * rec) +
               ((((static_cast<size_t>(F) * ((T / PL) + 1)) + 1) & ~size_t{1}) * 2) + (F * 4ull);
    };
    // one wave of resident CTAs is the target
    int occ = 0;
    allow_smem(fn);
    check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, static_cast<int>(T), smem_of(1)),
          "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    uint32_t const target = static_cast<uint32_t>(std::max(occ, 1)) * k_sms;
    // path lanes per row: raised until the row tiles fill the wave, or one row
    uint32_t lane_shift = 0;
    while ((1u << lane_shift) < T && ceil_div(n, T >> lane_shift) < target)
    {
        ++lane_shift;
    }
    uint32_t const PL       = 1u << lane_shift;
    uint32_t const rpb      = T >> lane_shift;
    uint32_t const row_blks = ceil_div(n, rpb);
    uint32_t const chunk    = chunk_of(PL);
    // split the paths when the row tiles still leave the wave short, each
    // lane keeping at least eight paths per split
    uint32_t splits = 1;
    if (row_blks < target)
    {
        uint32_t const most = std::max<uint32_t>(1, pl.n_paths / (8 * PL));
        splits              = std::min(ceil_div(target, row_blks), most);
        size_t const per    = n * (static_cast<size_t>(F) + 1) * sizeof(double);
        splits = static_cast<uint32_t>(
            std::min<size_t>(splits, std::max<size_t>(1, k_max_ws_bytes / per)));
    }
    uint32_t const pps = ceil_div(ceil_div(pl.n_paths, splits), chunk) * chunk;
    splits             = ceil_div(pl.n_paths, pps);
    size_t const smem  = smem_of(PL);
    double      *ws    = nullptr;
    if (splits > 1)
    {
        pl.ws.grow(static_cast<size_t>(splits) * n * (F + 1) * sizeof(double), pl.ws_cap);
        ws = pl.ws.as<double>();
    }
    dim3 const grid(row_blks, splits);
    fn<<<grid, T, smem, s>>>(p.u8 ? static_cast<uint8_t const *>(p.bins) : nullptr,
                             p.u8 ? nullptr : static_cast<uint16_t const *>(p.bins), p.n_pad,
                             n, pl.last.as<uint32_t>(), F, pl.heads.as<PathHead>(),
                             pl.elems.as<PathElem>(), pl.n_paths, pps, chunk, lane_shift,
                             pl.gauss, pl.lr, pl.bias, pl.init, splits > 1 ? nullptr : out, ws);
    check(cudaGetLastError(), "shap_tile_kernel");
    if (splits == 1)
    {
        return 1;
    }
    uint64_t const cells = n * (F + 1);
    shap_reduce_kernel<<<ceil_div(cells, 256), 256, 0, s>>>(ws, n, F, splits, pl.lr, pl.bias,
                                                           pl.init, out);
    check(cudaGetLastError(), "shap_reduce_kernel");
    return 2;
}

void shap_run_host(bb_shap_plan &pl, Plane const &p, double *out)
{
    std::lock_guard<std::mutex> lock(pl.mu);
    size_t const bytes = p.n_rows * (pl.n_feats + 1ull) * sizeof(double);
    if (bytes == 0)
    {
        return;
    }
    pl.out.grow(bytes, pl.out_cap);
    shap_launch(pl, p, pl.out.as<double>(), pl.stream);
    check(cudaMemcpyAsync(out, pl.out.p, bytes, cudaMemcpyDeviceToHost, pl.stream),
          "cudaMemcpyAsync");
    check(cudaStreamSynchronize(pl.stream), "cudaStreamSynchronize");
}

template <typename F> int shap_guard(F &&f)
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

} // namespace
} // namespace bb

using namespace bb;

extern "C"
{
    int bb_shap_plan_create(bb_plane const *plane, uint32_t n_trees, uint32_t const *roots,
                            uint32_t n_nodes, uint32_t const *feature, uint32_t const *split_bin,
                            uint32_t const *left, uint32_t const *right,
                            uint8_t const *default_left, float const *value, float const *cover,
                            float lr, float init, bb_shap_plan **out)
    {
        return shap_guard(
            [&]
            {
                if (plane == nullptr || out == nullptr)
                {
                    throw std::invalid_argument("bb_shap_plan_create: null argument");
                }
                *out = make_shap_plan(plane->p, n_trees, roots, n_nodes, feature, split_bin,
                                      left, right, default_left, value, cover, lr, init)
                           .release();
            });
    }

    int bb_shap_plan_run(bb_shap_plan *plan, bb_plane const *plane, double *out)
    {
        return shap_guard(
            [&]
            {
                if (plan == nullptr || plane == nullptr || out == nullptr)
                {
                    throw std::invalid_argument("bb_shap_plan_run: null argument");
                }
                shap_check_plane(*plan, plane->p);
                shap_run_host(*plan, plane->p, out);
            });
    }

    int bb_shap_plan_launch(bb_shap_plan *plan, bb_plane const *plane, double *out_device,
                            void *stream, uint32_t *launches)
    {
        return shap_guard(
            [&]
            {
                if (plan == nullptr || plane == nullptr || out_device == nullptr)
                {
                    throw std::invalid_argument("bb_shap_plan_launch: null argument");
                }
                shap_check_plane(*plan, plane->p);
                std::lock_guard<std::mutex> lock(plan->mu);
                uint32_t const k = shap_launch(*plan, plane->p, out_device,
                                               static_cast<cudaStream_t>(stream));
                if (launches != nullptr)
                {
                    *launches = k;
                }
            });
    }

    void bb_shap_plan_destroy(bb_shap_plan *plan)
    {
        delete plan;
    }

    int bb_pred_contribs(bb_plane const *plane, uint32_t n_trees, uint32_t const *roots,
                         uint32_t n_nodes, uint32_t const *feature, uint32_t const *split_bin,
                         uint32_t const *left, uint32_t const *right,
                         uint8_t const *default_left, float const *value, float const *cover,
                         float lr, float init, double *out)
    {
        return shap_guard(
            [&]
            {
                if (plane == nullptr || out == nullptr)
                {
                    throw std::invalid_argument("bb_pred_contribs: null argument");
                }
                auto pl = make_shap_plan(plane->p, n_trees, roots, n_nodes, feature, split_bin,
                                         left, right, default_left, value, cover, lr, init);
                shap_check_plane(*pl, plane->p);
                shap_run_host(*pl, plane->p, out);
            });
    }
}
