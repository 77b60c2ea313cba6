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
#include "nkb_dynamics.cuh"

namespace nkb {

constexpr int kTreeBase = 6;            // columns of a floating base

// This lane's place in the tree: its joint coordinate (lane, or lane + 32 on the base's lanes of a wide articulation), the
// number of ancestor joints, the lanes of its descendants, its ancestors' coordinates by depth, one byte each.
struct TreeLane {
    uint32_t coord, level, desc;
    uint32_t anc[kTreeLevels / 4];
    NKB_DEV uint32_t ancestor(int p) const { return (anc[p >> 2] >> (8 * (p & 3))) & 0xffu; }
};
constexpr uint32_t kTreeNone = 0xffu;   // level of a lane without a joint coordinate

NKB_DEV TreeLane tree_lane(const Env& e) {
    TreeLane t;
    const uint32_t* w = e.t->tree_lanes + e.lane * kTreeLaneWords;
    const uint32_t head = __ldg(w);
    t.coord = head & 0xffu; t.level = (head >> 8) & 0xffu;
    t.desc = __ldg(w + 1);
#pragma unroll
    for (int k = 0; k < kTreeLevels / 4; ++k) t.anc[k] = __ldg(w + 2 + k);
    return t;
}

// A lane's compressed row.
struct TreeRow {
    float base[kTreeBase], limb[kTreeLevels], diag;
};

// Row of the lane's coordinate out of a dense symmetric matrix in shared memory (rows of `ld` words, 16-byte aligned).
NKB_DEV void tree_load_row(const Env& e, const TreeLane& t, const float* matrix, uint32_t ld, TreeRow& row) {
    const float* src = matrix + t.coord * ld;
#pragma unroll
    for (int k = 0; k < kTreeBase; ++k) row.base[k] = 0.f;
    if (e.t->floating_root) {
        const float4 lo = *reinterpret_cast<const float4*>(src);
        const float2 hi = *reinterpret_cast<const float2*>(src + 4);
        row.base[0] = lo.x; row.base[1] = lo.y; row.base[2] = lo.z; row.base[3] = lo.w; row.base[4] = hi.x; row.base[5] = hi.y;
    }
    const int depth = (int)e.t->tree_depth;
#pragma unroll
    for (int p = 0; p < kTreeLevels; ++p) row.limb[p] = 0.f;
#pragma unroll
    for (int p = 0; p < kTreeLevels; p += 2) {
        if (p >= depth - 1) break;
        row.limb[p] = src[t.ancestor(p)]; row.limb[p + 1] = src[t.ancestor(p + 1)];
    }
    row.diag = src[t.coord];
}

// Solves A x = g.  `row` and `g` are the joint lanes' rows and right-hand sides; lanes 0..5 carry the base's rows in
// `base_row` (lower triangle) and its right-hand sides in `base_g`.  `scratch` holds tree_scratch_words.  On return `x` is the
// joint lanes' solution and `base_x` (every lane) the base's.  False when a pivot is not positive and finite.
template <int NR>
NKB_DEV bool tree_solve(const Env& e, const TreeLane& t, TreeRow& row, float g, const float (&base_row)[kTreeBase], float base_g,
                        float* scratch, float& x, float (&base_x)[kTreeBase]) {
    const uint32_t stride = e.t->tree_stride, lane = e.lane;
    const int depth = (int)e.t->tree_depth;
    // rows are indexed by joint lane; with one coordinate per lane the base's lanes hold no joint and get no row
    const uint32_t first = NR == 1 && e.t->floating_root ? 6u : 0u, rows = NR == 1 ? e.t->ndof - first : 32u;
    float* mine = scratch + (lane - first) * stride;
    float inverse = 1.f, y = 0.f;
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
            valid = row.diag > 0.f && row.diag <= FLT_MAX;
            inverse = rsqrtf(valid ? row.diag : 1.0f);
            y = g * inverse;
#pragma unroll
            for (int k = 0; k < kTreeBase; ++k) row.base[k] *= inverse;
            float4* out = reinterpret_cast<float4*>(mine);
            out[0] = make_float4(row.base[0], row.base[1], row.base[2], row.base[3]);
            out[1] = make_float4(row.base[4], row.base[5], y, 0.f);
#pragma unroll
            for (int k = 0; k < kTreeLevels; k += 4) {
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
            g = fmaf(-m, b1.z, g);
#pragma unroll
            for (int q = 0; q < kTreeLevels; q += 4) {
                if (q >= 4 * quads) break;
                const float4 c4 = *reinterpret_cast<const float4*>(src + 8 + q);
                row.limb[q] = fmaf(-m, c4.x, row.limb[q]); row.limb[q + 1] = fmaf(-m, c4.y, row.limb[q + 1]);
                row.limb[q + 2] = fmaf(-m, c4.z, row.limb[q + 2]); row.limb[q + 3] = fmaf(-m, c4.w, row.limb[q + 3]);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < kTreeBase; ++k) base_x[k] = 0.f;
    float acc = y;
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
            float s0 = block[8u * i + j], s1 = 0.f;
            const float* src = scratch;
            uint32_t k = 0u;
#pragma unroll 1
            for (; k + 1u < rows; k += 2u, src += 2u * stride) {
                s0 = fmaf(-src[i], src[j], s0);
                s1 = fmaf(-src[stride + i], src[stride + j], s1);
            }
            if (k < rows) s0 = fmaf(-src[i], src[j], s0);
            entries[lane] = s0 + s1;
        }
        __syncwarp();
        float a[28];
#pragma unroll
        for (int k = 0; k < 7; ++k) { const float4 v = reinterpret_cast<const float4*>(entries)[k]; a[4 * k] = v.x; a[4 * k + 1] = v.y; a[4 * k + 2] = v.z; a[4 * k + 3] = v.w; }
        float inv[kTreeBase];
#pragma unroll
        for (int k = 0; k < kTreeBase; ++k) {
            const float pivot = a[k * (k + 1) / 2 + k];
            const bool good = pivot > 0.f && pivot <= FLT_MAX;
            valid &= good;
            inv[k] = rsqrtf(good ? pivot : 1.0f);
            a[21 + k] *= inv[k];
#pragma unroll
            for (int i = k + 1; i < kTreeBase; ++i) a[i * (i + 1) / 2 + k] *= inv[k];
#pragma unroll
            for (int i = k + 1; i < kTreeBase; ++i) {
                a[21 + i] = fmaf(-a[i * (i + 1) / 2 + k], a[21 + k], a[21 + i]);
#pragma unroll
                for (int j = k + 1; j <= i; ++j) a[i * (i + 1) / 2 + j] = fmaf(-a[i * (i + 1) / 2 + k], a[j * (j + 1) / 2 + k], a[i * (i + 1) / 2 + j]);
            }
        }
#pragma unroll
        for (int k = kTreeBase - 1; k >= 0; --k) {
            float s = a[21 + k];
#pragma unroll
            for (int i = k + 1; i < kTreeBase; ++i) s = fmaf(-a[i * (i + 1) / 2 + k], base_x[i], s);
            base_x[k] = s * inv[k];
        }
#pragma unroll
        for (int k = 0; k < kTreeBase; ++k) acc = fmaf(-row.base[k], base_x[k], acc);
    }
    if (!__all_sync(NKB_FULL, valid)) return false;
    // joints root to leaf: a depth's solution reaches its descendants by shuffle
#pragma unroll
    for (int p = 0; p < kTreeLevels - 1; ++p) {
        if (p >= depth - 1) break;
        const float xp = __shfl_sync(NKB_FULL, acc * inverse, t.ancestor(p) & 31u);
        if (t.level != kTreeNone && t.level > (uint32_t)p) acc = fmaf(-row.limb[p], xp, acc);
    }
    x = acc * inverse;
    return true;
}

}  // namespace nkb
