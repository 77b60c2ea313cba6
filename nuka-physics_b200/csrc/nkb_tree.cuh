// Factorisation and solve of a symmetric positive matrix with the sparsity of the articulation's tree, by one warp.
//
// Entry (i, k) of the mass matrix, and of J^T C J for constraint rows that act along a single root path, is zero unless one
// coordinate is an ancestor of the other.  Eliminating leaves first keeps that pattern (no fill-in), and all coordinates of
// one depth are pivots at the same time, so the serial chain is as long as the tree is deep (3 for a quadruped's legs, 10
// for a humanoid's arms behind its waist) instead of as long as the matrix is wide (18, 35).
//
// A lane owns the row of one joint coordinate, compressed to the columns it can be nonzero in: the floating base's six, then
// one per ancestor joint, by depth.  Columns are static register indices because the depth, not the coordinate, names
// them.  The base's own 6 x 6 block is the Schur complement left when all joints are eliminated: one lane per entry sums
// the joints' contributions, then every lane factors the block in registers for itself (no exchange inside the chain).
//
// A pivot lane publishes its scaled row in shared memory, 8 words (base columns, solved right-hand side) plus the limb
// columns; the ancestors of that depth pull their multiplier and the row from there.  Row strides of 12 and 20 words keep
// float4 reads of different rows free of bank conflicts.
#pragma once
#include <type_traits>
#include "nkb_env.cuh"

namespace nkb {

constexpr int kTreeBase = 6;            // columns of a floating base

// This lane's place in the tree: its joint coordinate (lane, or lane + 32 on the base's lanes of a wide articulation), the
// number of ancestor joints, the lanes of its descendants, its ancestors' coordinates by depth, one byte each; and the tree's depth and
// row stride in shared memory.
template <int kLevels>
struct TreeLane {
    uint32_t coord, level, desc, depth, stride;
    uint32_t anc[kLevels / 4];
    NKB_DEV uint32_t ancestor(int p) const { return (anc[p >> 2] >> (8 * (p & 3))) & 0xffu; }
    // the same where p is no constant
    NKB_DEV uint32_t ancestor_at(int p) const {
        uint32_t word = anc[0];
#pragma unroll
        for (int k = 1; k < kLevels / 4; ++k) if (p >= 4 * k) word = anc[k];
        return (word >> (8 * (p & 3))) & 0xffu;
    }
};
constexpr uint32_t kTreeNone = 0xffu;   // level of a lane without a joint coordinate

template <int kLevels = kTreeLevels>
NKB_DEV TreeLane<kLevels> tree_lane(const Env& e) {
    TreeLane<kLevels> t;
    const uint32_t* w = e.t->tree_lanes + e.lane * kTreeLaneWords;
    const uint32_t head = __ldg(w);
    t.coord = head & 0xffu; t.level = (head >> 8) & 0xffu;
    t.desc = __ldg(w + 1);
    t.depth = e.t->tree_depth; t.stride = e.t->tree_stride;
#pragma unroll
    for (int k = 0; k < kLevels / 4; ++k) t.anc[k] = k < kTreeLevels / 4 ? __ldg(w + 2 + k) : 0u;
    return t;
}
// The same in the tree that merge_trees left.
template <int kLevels>
NKB_DEV TreeLane<kLevels> merged_lane(const Env& e) {
    TreeLane<kLevels> t;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(e.sm + e.lay->merged) + e.lane * merged_lane_words(e.t->ndof);
    t.coord = w[0] & 0xffu; t.level = (w[0] >> 8) & 0xffu;
    t.desc = w[1];
    t.depth = e.merged; t.stride = tree_row_stride(e.merged);
#pragma unroll
    for (int k = 0; k < kLevels / 4; ++k) t.anc[k] = w[2 + k];
    return t;
}

// A lane's compressed row.
template <int kLevels>
struct TreeRow {
    float base[kTreeBase], limb[kLevels], diag;
};

// Row of the lane's coordinate out of a dense symmetric matrix in shared memory (rows of `ld` words, 16-byte aligned).
template <int kLevels>
NKB_DEV void tree_load_row(const Env& e, const TreeLane<kLevels>& t, const float* matrix, uint32_t ld, TreeRow<kLevels>& row) {
    const float* src = matrix + t.coord * ld;
#pragma unroll
    for (int k = 0; k < kTreeBase; ++k) row.base[k] = 0.f;
    if (e.t->floating_root) {
        const float4 lo = *reinterpret_cast<const float4*>(src);
        const float2 hi = *reinterpret_cast<const float2*>(src + 4);
        row.base[0] = lo.x; row.base[1] = lo.y; row.base[2] = lo.z; row.base[3] = lo.w; row.base[4] = hi.x; row.base[5] = hi.y;
    }
    const int depth = (int)t.depth;
#pragma unroll
    for (int p = 0; p < kLevels; ++p) row.limb[p] = 0.f;
#pragma unroll
    for (int p = 0; p < kLevels; p += 2) {
        if (p >= depth - 1) break;
        row.limb[p] = src[t.ancestor(p)]; row.limb[p + 1] = src[t.ancestor(p + 1)];
    }
    row.diag = src[t.coord];
}

// Rows of the tree in shared memory: joint lanes first .. first + rows.  With one coordinate per lane the base's lanes hold no
// joint and get no row.
template <int NR> NKB_DEV uint32_t tree_first(const Env& e) { return NR == 1 && e.t->floating_root ? 6u : 0u; }
template <int NR> NKB_DEV uint32_t tree_rows(const Env& e) { return NR == 1 ? e.t->ndof - tree_first<NR>(e) : 32u; }

// Solves A x = rhs.  `row` and `rhs` are the joint lanes' rows and right-hand sides; lanes 0..5 carry the base's rows in
// `base_row` (lower triangle) and its right-hand sides in `base_g`.  `scratch` holds tree_scratch_words.  On return `x` is the
// joint lanes' solution and `base_x` (every lane) the base's.  False when a pivot is not positive and finite.
// kKeep leaves the factor in `scratch` for tree_mass_solve and tree_coupling: the scaled rows with their reciprocal pivot roots
// in word 7, the base block's triangle and reciprocal roots in the 28 words behind the base rows; pivots are held to the mass
// matrix's floor.  It serves the joint accelerations, so it rounds correctly where the Newton systems approximate, and sums the
// right-hand side and the base's Schur complement in 64 bits: eliminated last, the base gathers the cancellations of all limbs.
// M^-1 tau against 64 bits, root mean square over 2048 humanoids: 8.0e-7 with approximate roots and 32-bit sums, 5.0e-7 so (the
// dense factor, base first, 5.1e-7); quadrupeds 1.35e-7 and 0.86e-7 (dense 1.5e-7).  It costs their policy steps 0.7 %.
template <int NR, bool kKeep, int kLevels>
NKB_DEV bool tree_solve(const Env& e, const TreeLane<kLevels>& t, TreeRow<kLevels>& row, float rhs, const float (&base_row)[kTreeBase], float base_g,
                        float* scratch, float& x, float (&base_x)[kTreeBase]) {
    const uint32_t stride = t.stride, lane = e.lane;
    const int depth = (int)t.depth;
    const uint32_t first = tree_first<NR>(e), rows = tree_rows<NR>(e);
    float* mine = scratch + (lane - first) * stride;
    using Sum = typename std::conditional<kKeep, double, float>::type;
    Sum g = rhs;
    float inverse = 1.f;
    Sum y = 0.f;
    bool valid = true;
    if (NR > 1 && t.level == kTreeNone) {            // a lane without a joint between others: contributes zero to the base
        reinterpret_cast<float4*>(mine)[0] = make_float4(0.f, 0.f, 0.f, 0.f);
        reinterpret_cast<float4*>(mine)[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // depths leaf to root; the loop is rolled and the limb columns go in fours (columns at or past a lane's own depth hold
    // values nothing reads), which keeps the routine at a few KB of instructions
    const int quads = (depth + 2) >> 2;             // groups of four limb columns in use
#pragma unroll 1
    for (int p = depth - 1; p >= 0; --p) {
        const uint32_t pivots = __ballot_sync(NKB_FULL, t.level == (uint32_t)p);
        if (t.level == (uint32_t)p) {
            if (kKeep) row.diag = fmaxf(row.diag, kMassPivotFloor);
            valid = pivot_valid(row.diag);
            inverse = kKeep ? __frsqrt_rn(row.diag) : rsqrt_normal(row.diag);
            y = g * inverse;
#pragma unroll
            for (int k = 0; k < kTreeBase; ++k) row.base[k] *= inverse;
            float4* out = reinterpret_cast<float4*>(mine);
            out[0] = make_float4(row.base[0], row.base[1], row.base[2], row.base[3]);
            out[1] = make_float4(row.base[4], row.base[5], (float)y, inverse);
#pragma unroll
            for (int k = 0; k < kLevels; k += 4) {
                if (k >= 4 * quads) break;
#pragma unroll
                for (int c = 0; c < 4; ++c) row.limb[k + c] *= inverse;
                out[2 + (k >> 2)] = make_float4(row.limb[k], row.limb[k + 1], row.limb[k + 2], row.limb[k + 3]);
            }
        }
        __syncwarp();
        // ancestors of this depth's pivots pull their updates
        uint32_t below = t.level < (uint32_t)p ? (t.desc & pivots) : 0u;
#pragma unroll 1
        while (below != 0u) {
            const uint32_t k = (uint32_t)__ffs(below) - 1u;
            below &= below - 1u;
            const float* src = scratch + (k - first) * stride;
            const float m = src[8u + t.level];
            const float4 b0 = *reinterpret_cast<const float4*>(src), b1 = *reinterpret_cast<const float4*>(src + 4);
            row.diag = fmaf(-m, m, row.diag);
            row.base[0] = fmaf(-m, b0.x, row.base[0]); row.base[1] = fmaf(-m, b0.y, row.base[1]); row.base[2] = fmaf(-m, b0.z, row.base[2]);
            row.base[3] = fmaf(-m, b0.w, row.base[3]); row.base[4] = fmaf(-m, b1.x, row.base[4]); row.base[5] = fmaf(-m, b1.y, row.base[5]);
            g = fma((Sum)-m, (Sum)b1.z, g);
#pragma unroll
            for (int q = 0; q < kLevels; q += 4) {
                if (q >= 4 * quads) break;
                const float4 c4 = *reinterpret_cast<const float4*>(src + 8 + q);
                row.limb[q] = fmaf(-m, c4.x, row.limb[q]); row.limb[q + 1] = fmaf(-m, c4.y, row.limb[q + 1]);
                row.limb[q + 2] = fmaf(-m, c4.z, row.limb[q + 2]); row.limb[q + 3] = fmaf(-m, c4.w, row.limb[q + 3]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kTreeBase; ++k) base_x[k] = 0.f;
    Sum acc = y;
    if (e.t->floating_root) {
        // Schur complement of the base, lane = entry (21 of the lower triangle, then the 6 right-hand sides)
        float* block = scratch + rows * stride;                      // 6 x 8 base rows, then 28 entries
        if (lane < 6u) {
            float4* out = reinterpret_cast<float4*>(block + 8u * lane);
            out[0] = make_float4(base_row[0], base_row[1], base_row[2], base_row[3]);
            out[1] = make_float4(base_row[4], base_row[5], base_g, 0.f);
        }
        __syncwarp();
        float* entries = block + 48;
        if (lane < 27u) {
            // entry -> (row i, column j): i(i+1)/2 + j for the triangle
            uint32_t i, j;
            if (lane >= 21u) { i = lane - 21u; j = 6u; }
            else { i = lane >= 15u ? 5u : lane >= 10u ? 4u : lane >= 6u ? 3u : lane >= 3u ? 2u : lane >= 1u ? 1u : 0u; j = lane - (i * (i + 1u)) / 2u; }
            // Two chains, the base's own entry last: the joints' terms nearly cancel it.  On systems of this kind (20 000 random ones of
            // 12 joints and of 29) 32-bit sums are off by 1.02e-7 and 1.34e-7 (root mean square, of the base's entries), in two chains
            // that begin with it by 1.18e-7 and 1.62e-7, in one by 1.15e-7 and 1.67e-7.  A landing quadruped's trajectory tells any two
            // roundings apart: the second form misses the reference's bars in one env of one case, as 64-bit sums do.
            Sum s0 = 0.f, s1 = 0.f;
            const float* src = scratch;
            uint32_t k = 0u;
#pragma unroll 1
            for (; k + 1u < rows; k += 2u, src += 2u * stride) {
                s0 = fma((Sum)-src[i], (Sum)src[j], s0);
                s1 = fma((Sum)-src[stride + i], (Sum)src[stride + j], s1);
            }
            if (k < rows) s0 = fma((Sum)-src[i], (Sum)src[j], s0);
            s0 = (s0 + s1) + (Sum)block[8u * i + j];
            if (kKeep && j == 6u) *reinterpret_cast<double*>(block + 8u * i + 6u) = s0;        // in place of base_g and its pad
            else entries[lane] = (float)(s0);
        }
        __syncwarp();
        float packed[28], a[21];
        Sum z[kTreeBase];
#pragma unroll
        for (int k = 0; k < 7; ++k) { const float4 v = reinterpret_cast<const float4*>(entries)[k]; packed[4 * k] = v.x; packed[4 * k + 1] = v.y; packed[4 * k + 2] = v.z; packed[4 * k + 3] = v.w; }
#pragma unroll
        for (int k = 0; k < 21; ++k) a[k] = packed[k];
#pragma unroll
        for (int k = 0; k < kTreeBase; ++k) z[k] = kKeep ? (Sum)*reinterpret_cast<const double*>(block + 8 * k + 6) : (Sum)packed[21 + k];
        if (kKeep) __syncwarp();
        float inv[kTreeBase];
        valid &= solve6<kKeep>(a, z, inv, base_x);
        if (kKeep && lane == 0u) {          // every lane holds the block; nobody reads the entries any more
            float4* out = reinterpret_cast<float4*>(entries);
#pragma unroll
            for (int k = 0; k < 5; ++k) out[k] = make_float4(a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3]);
            out[5] = make_float4(a[20], inv[0], inv[1], inv[2]);
            out[6] = make_float4(inv[3], inv[4], inv[5], 0.f);
        }
#pragma unroll
        for (int k = 0; k < kTreeBase; ++k) acc = fma((Sum)-row.base[k], (Sum)base_x[k], acc);
    }
    if (!kKeep && !__all_sync(NKB_FULL, valid)) return false;
    // joints root to leaf: a depth's solution reaches its descendants by shuffle
#pragma unroll 1
    for (int p = 0; p < depth - 1; ++p) {
        const float xp = __shfl_sync(NKB_FULL, (float)(acc * inverse), t.ancestor_at(p) & 31u);
        if (t.level != kTreeNone && t.level > (uint32_t)p) acc = fma((Sum)-mine[8 + p], (Sum)xp, acc);
    }
    x = (float)(acc * inverse);
    return true;
}

// Spreads a solution over the lanes' coordinates: joints from their lanes, the base's from the replicated copy.
template <int NR>
NKB_DEV void tree_scatter(const Env& e, float joint, const float (&base_x)[kTreeBase], float (&x)[NR]) {
    const uint32_t l = e.lane, n = e.t->ndof;
    if (e.t->floating_root && l < 6u) {
        if (NR > 1) x[NR - 1] = l + 32u < n ? joint : 0.f;
        x[0] = l == 0u ? base_x[0] : l == 1u ? base_x[1] : l == 2u ? base_x[2] : l == 3u ? base_x[3] : l == 4u ? base_x[4] : base_x[5];
    } else {
        if (NR > 1) x[NR - 1] = 0.f;
        x[0] = l < n ? joint : 0.f;
    }
}

// x = M^-1 g with the kept factor: g and x are the joint lanes' entries, base_g / base_x the base's (lane k of the first six
// carries base_g of coordinate k; base_x in every lane).
template <int NR>
NKB_DEV void tree_mass_solve(const Env& e, const TreeLane<kTreeLevels>& t, float* factor, float g, float base_g, float& x, float (&base_x)[kTreeBase]) {
    const uint32_t stride = e.t->tree_stride, lane = e.lane, first = tree_first<NR>(e), rows = tree_rows<NR>(e);
    const int depth = (int)e.t->tree_depth;
    const bool joint = t.level != kTreeNone;
    float* mine = factor + (joint ? lane - first : 0u) * stride;
    const float inverse = joint ? mine[7] : 1.f;
    float y = 0.f;
    __syncwarp();
#pragma unroll 1
    for (int p = depth - 1; p >= 0; --p) {
        const uint32_t pivots = __ballot_sync(NKB_FULL, t.level == (uint32_t)p);
        if (t.level == (uint32_t)p) { y = g * inverse; mine[6] = y; }
        __syncwarp();
        uint32_t below = t.level < (uint32_t)p ? (t.desc & pivots) : 0u;
#pragma unroll 1
        while (below != 0u) {
            const float* src = factor + ((uint32_t)__ffs(below) - 1u - first) * stride;
            below &= below - 1u;
            g = fmaf(-src[8u + t.level], src[6], g);
        }
    }
#pragma unroll
    for (int k = 0; k < kTreeBase; ++k) base_x[k] = 0.f;
    float acc = y;
    if (e.t->floating_root) {
        float* block = factor + rows * stride;
        if (lane < 6u) {
            const float* src = factor;
            float s = base_g;
#pragma unroll 1
            for (uint32_t k = 0u; k < rows; ++k, src += stride) s = fmaf(-src[lane], src[6], s);
            block[lane] = s;
        }
        __syncwarp();
        float a[28], z[8];
#pragma unroll
        for (int k = 0; k < 7; ++k) { const float4 v = reinterpret_cast<const float4*>(block + 48)[k]; a[4 * k] = v.x; a[4 * k + 1] = v.y; a[4 * k + 2] = v.z; a[4 * k + 3] = v.w; }
#pragma unroll
        for (int k = 0; k < 2; ++k) { const float4 v = reinterpret_cast<const float4*>(block)[k]; z[4 * k] = v.x; z[4 * k + 1] = v.y; z[4 * k + 2] = v.z; z[4 * k + 3] = v.w; }
#pragma unroll
        for (int k = 0; k < kTreeBase; ++k) {
            z[k] *= a[21 + k];
#pragma unroll
            for (int i = k + 1; i < kTreeBase; ++i) z[i] = fmaf(-a[i * (i + 1) / 2 + k], z[k], z[i]);
        }
#pragma unroll
        for (int k = kTreeBase - 1; k >= 0; --k) {
            base_x[k] = z[k] * a[21 + k];
#pragma unroll
            for (int i = 0; i < k; ++i) z[i] = fmaf(-a[k * (k + 1) / 2 + i], base_x[k], z[i]);
        }
        const float4 b0 = reinterpret_cast<const float4*>(mine)[0];
        const float2 b1 = reinterpret_cast<const float2*>(mine)[2];
        acc = fmaf(-b0.x, base_x[0], acc); acc = fmaf(-b0.y, base_x[1], acc); acc = fmaf(-b0.z, base_x[2], acc);
        acc = fmaf(-b0.w, base_x[3], acc); acc = fmaf(-b1.x, base_x[4], acc); acc = fmaf(-b1.y, base_x[5], acc);
    }
#pragma unroll 1
    for (int p = 0; p < depth - 1; ++p) {
        const float xp = __shfl_sync(NKB_FULL, acc * inverse, t.ancestor_at(p) & 31u);
        if (joint && t.level > (uint32_t)p) acc = fmaf(-mine[8 + p], xp, acc);
    }
    x = acc * inverse;
}

// J M^-1 J^T = |L^-1 J^T|^2 of one row per lane, for rows that act on the base and along one root path: `row` is the row's
// dense entries (or null for a row with the single entry `unit` at coordinate `leaf`), `leaf` the deepest coordinate of its
// path (0xff: the base alone).  The forward solve only touches the path and the base, so lanes work on rows of their own.
template <int NR>
NKB_DEV float tree_coupling(const Env& e, const float* factor, const float* row, uint32_t leaf, float unit) {
    const uint32_t stride = e.t->tree_stride, first = tree_first<NR>(e), rows = tree_rows<NR>(e);
    float z[kTreeBase], total = 0.f;
    const bool floating = e.t->floating_root != 0u;
#pragma unroll
    for (int k = 0; k < kTreeBase; ++k) z[k] = row != nullptr && floating ? row[k] : 0.f;
    if (leaf != 0xffu) {
        const uint32_t* table = e.t->tree_lanes + (leaf & 31u) * kTreeLaneWords;
        const int level = (int)((__ldg(table) >> 8) & 0xffu);
        float path[kTreeLevels];                             // remaining right-hand side along the path
#pragma unroll
        for (int p = 0; p < kTreeLevels; ++p) {
            path[p] = 0.f;
            if (row != nullptr && p < level) path[p] = row[(__ldg(table + 2 + (p >> 2)) >> (8 * (p & 3))) & 0xffu];
        }
        float g = row != nullptr ? row[leaf] : unit;
        uint32_t at = leaf;
#pragma unroll 1
        for (int p = level; p >= 0; --p) {
            const float* src = factor + ((at & 31u) - first) * stride;
            const float y = g * src[7];
            total = fmaf(y, y, total);
#pragma unroll
            for (int k = 0; k < kTreeBase; ++k) z[k] = fmaf(-src[k], y, z[k]);
            g = 0.f;
#pragma unroll
            for (int q = 0; q < kTreeLevels - 1; ++q)
                if (q < p) { path[q] = fmaf(-src[8 + q], y, path[q]); if (q == p - 1) g = path[q]; }
            if (p > 0) at = (__ldg(table + 2 + ((p - 1) >> 2)) >> (8 * ((p - 1) & 3))) & 0xffu;
        }
    }
    if (floating) {
        const float* a = factor + rows * stride + 48;
#pragma unroll
        for (int k = 0; k < kTreeBase; ++k) {
            z[k] *= a[21 + k];
            total = fmaf(z[k], z[k], total);
#pragma unroll
            for (int i = k + 1; i < kTreeBase; ++i) z[i] = fmaf(-a[i * (i + 1) / 2 + k], z[k], z[i]);
        }
    }
    return total;
}

}  // namespace nkb
