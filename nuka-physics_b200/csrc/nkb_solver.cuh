// Warp-per-env block-descent velocity solve with split-impulse position pass.
// Blocks are the env's free bodies (6 coordinates: linear, angular) followed by its articulation (one
// coordinate per DoF).  Blocks descend colour by colour; each block takes safeguarded Newton steps with an
// exact line search on its local augmented Lagrangian, then the multipliers update with momentum.
// One lane owns one block coordinate in the Newton system and one head in the row evaluations.
// The algorithm is that of the reference's tile route: ops/block_descent_tile.cuh:743-797 (head setup),
// :1103-1144 (colouring), :1508-1666 (assemble/factor/solve), :2089-2301 (line search, block descent),
// :2493-2595 (dual update), :2379-2489 (momentum balance), :2608-2744 (finish, position marks),
// :2942-3087 (sweep loop) and ops/block_descent.cu:1734-1753 (position bias).
#pragma once
#include "nkb_rowspace.cuh"

namespace nkb {

static_assert(HF_COUNT == kHeadStride, "head record must match the host layout");

constexpr uint32_t kNewtonSteps = 16u, kLineSteps = 32u;
constexpr float kLineTol = 1.0e-6f, kRoundings = 8.0f;
// An impulse is rho (residual - move) + multiplier, so its own rounding error, half an ulp each of the move, the difference
// and the sum, scales with those terms even where they cancel: up to eps (|f| + rho (|residual| + |move|)).  The line search
// accepts a slope below that bound once (kRoundings x this factor = 1): nothing smaller can be told from zero.  With |f| alone
// in the bound one search in six ended below the noise and above the bound, and halved its interval down to the last bit
// (26 evaluations instead of 1 to 3).
constexpr float kImpulseRounding = 1.0f / kRoundings;

struct Tile {
    uint32_t nheads, nblocks;
    bool units;                         // there are rows on a single coordinate
    float momentum, residual, tol;
};

NKB_DEV uint32_t* sm_binfo(const Env& e) { return reinterpret_cast<uint32_t*>(e.sm + e.lay->binfo); }
// binfo words: dim[nb], color[nb], inc_begin[nb + 1], inc[2 * head_cap], utab[3 * vstride, 16 bits each], order[nb + 1]
NKB_DEV uint32_t& blk_dim(const Env& e, uint32_t b) { return sm_binfo(e)[b]; }
NKB_DEV uint32_t& blk_color(const Env& e, uint32_t nb, uint32_t b) { return sm_binfo(e)[nb + b]; }
NKB_DEV uint32_t& blk_inc_begin(const Env& e, uint32_t nb, uint32_t b) { return sm_binfo(e)[2u * nb + b]; }
NKB_DEV uint32_t* blk_inc(const Env& e, uint32_t nb) { return sm_binfo(e) + 3u * nb + 1u; }
// unit rows of the articulation by coordinate: utab[slot * vstride + coordinate] = head or 0xffff (slots: lower limit,
// upper limit, dry friction; vstride = 32 or 64 coordinates), 16-bit entries
constexpr uint32_t kNoUnitHead = 0xffffu;
NKB_DEV uint16_t* unit_table(const Env& e, uint32_t nb) { return reinterpret_cast<uint16_t*>(sm_binfo(e) + 3u * nb + 1u + 2u * e.t->head_cap); }
// moving blocks in descent order, order[nb] = their count
NKB_DEV uint32_t* block_order(const Env& e, uint32_t nb) { return sm_binfo(e) + 3u * nb + 1u + 2u * e.t->head_cap + 3u * e.vstride / 2u; }
NKB_DEV float* sm_bmass(const Env& e, uint32_t b) { return e.sm + e.lay->bmass + 7u * free_slot(e, b); }
NKB_DEV float* sm_bfree(const Env& e, uint32_t b) { return e.sm + e.lay->bfree + 6u * free_slot(e, b); }
NKB_DEV float* sm_bpseudo(const Env& e, uint32_t b) { return e.sm + e.lay->bpseudo + 6u * free_slot(e, b); }

NKB_DEV uint32_t head_axes(const Env& e, uint32_t h) { return (hu(e, HF_FLAGS, h) & (kHeadContact | kHeadScalar)) == kHeadContact ? 3u : 1u; }
NKB_DEV uint32_t head_owner(const Env& e, uint32_t h, uint32_t side) { const uint32_t o = hu(e, HF_OWNER, h); return side == 0u ? (o & 0xffffu) : (o >> 16); }

// Jacobian entry of head h (incidence `side`) on coordinate i of its block, for contact axis ax.
NKB_DEV float head_jac(const Env& e, uint32_t h, uint32_t side, uint32_t ax, uint32_t i, uint32_t block) {
    const TemplateView& t = *e.t;
    if (block == t.B) {
        const uint32_t jo = hu(e, HF_JOFF, h);
        if (jo & kUnitRow) return i == (jo & 0xffffu) ? hf(e, HF_UNITV, h) : 0.f;
        return sm_jpool(e)[jo + ax * ((t.ndof + 3u) & ~3u) + i];
    }
    const V3 dir = hf3(e, ax == 0u ? HF_N : ax == 1u ? HF_T1 : HF_T2, h);
    const float sgn = side == 0u ? 1.f : -1.f;
    if (i < 3u) return sgn * comp(dir, (int)i);
    const V3 r = hf3(e, side == 0u ? HF_RA : HF_RB, h);
    return sgn * comp(cross(r, dir), (int)i - 3);
}

// J_h[ax] . u over the coordinates of block b (u padded with zeros to a multiple of 4 for the articulation).
NKB_DEV float head_row_dot(const Env& e, uint32_t h, uint32_t side, uint32_t ax, uint32_t block, const float* u) {
    const TemplateView& t = *e.t;
    if (block == t.B) {
        const uint32_t jo = hu(e, HF_JOFF, h);
        if (jo & kUnitRow) return hf(e, HF_UNITV, h) * u[jo & 0xffffu];
        const uint32_t chunks = (t.ndof + 3u) >> 2;
        const float4* j4 = reinterpret_cast<const float4*>(sm_jpool(e) + jo) + ax * chunks;
        const float4* u4 = reinterpret_cast<const float4*>(u);
        float s = 0.f;
#pragma unroll 1
        for (uint32_t c = 0u; c < chunks; ++c) {
            const float4 a = j4[c], b4 = u4[c];
            s = fmaf(a.x, b4.x, s); s = fmaf(a.y, b4.y, s); s = fmaf(a.z, b4.z, s); s = fmaf(a.w, b4.w, s);
        }
        return s;
    }
    float s = 0.f;
#pragma unroll 1
    for (uint32_t i = 0u; i < 6u; ++i) s += head_jac(e, h, side, ax, i, block) * u[i];
    return s;
}

NKB_DEV float* block_vel(const Env& e, uint32_t block, bool position) {
    if (block == e.t->B) return sm_vec(e, position ? kVecPseudo : kVecU);
    return position ? sm_bpseudo(e, block) : sm_bvel(e, block);
}
NKB_DEV const float* block_free(const Env& e, uint32_t block) { return block == e.t->B ? sm_vec(e, kVecFree) : sm_bfree(e, block); }

// x = M^-1 g for a block; a lane holds coordinates lane + 32 r.
template <int NR>
NKB_DEV void solve_block_mass(const Env& e, uint32_t block, const float (&g)[NR], float (&x)[NR]) {
    const TemplateView& t = *e.t;
    const uint32_t l = e.lane;
    if (block == t.B && t.mass_tree != 0u) {
        const bool high = NR > 1 && t.floating_root != 0u && l < 6u;
        float joint, base_x[kTreeBase];
        tree_mass_solve<NR>(e, tree_lane(e), sm_factor(e), high ? g[NR - 1] : g[0], g[0], joint, base_x);
        tree_scatter<NR>(e, joint, base_x, x);
        return;
    }
    if (block == t.B) {
        const uint32_t n = t.ndof, ld = e.lay->ld;
        const float* F = sm_factor(e);
#pragma unroll
        for (int r = 0; r < NR; ++r) x[r] = l + 32u * r < n ? g[r] : 0.f;
#pragma unroll 1
        for (uint32_t j = 0; j < n; ++j) {
            const float xj = coord_bcast<NR>(x, j);
#pragma unroll
            for (int r = 0; r < NR; ++r) { const uint32_t row = l + 32u * r; if (row > j && row < n) x[r] -= F[row * ld + j] * xj; }
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) { const uint32_t row = l + 32u * r; if (row < n) x[r] /= F[row * ld + row]; }
#pragma unroll 1
        for (uint32_t jj = n; jj > 0u; --jj) {
            const uint32_t j = jj - 1u;
            const float xj = coord_bcast<NR>(x, j);
#pragma unroll
            for (int r = 0; r < NR; ++r) { const uint32_t row = l + 32u * r; if (row < j) x[r] -= F[j * ld + row] * xj; }
        }
        return;
    }
    const float g3 = __shfl_sync(NKB_FULL, g[0], 3), g4 = __shfl_sync(NKB_FULL, g[0], 4), g5 = __shfl_sync(NKB_FULL, g[0], 5);
#pragma unroll
    for (int r = 0; r < NR; ++r) x[r] = 0.f;
    if (l < 3u) x[0] = g[0] * __ldg(t.inv_mass + block);
    else if (l < 6u) { const V3 w = sym_mulv(sm_bwinv(e, block), mk3(g3, g4, g5)); x[0] = comp(w, (int)l - 3); }
}

// J M^-1 J^T of an articulated row from one forward solve with the unit-lower factor (articulation_mass.cuh:413-441)
// Row with a single entry `value` at coordinate `at`: the solve starts there, the leading zeros contribute nothing.
template <int NR>
NKB_DEV float mass_coupling_unit(const Env& e, uint32_t at, float value) {
    const uint32_t n = e.t->ndof, ld = e.lay->ld;
    const float* F = sm_factor(e);
    float y[32 * NR];
    float r = 0.f;
#pragma unroll 1
    for (uint32_t i = at; i < n; ++i) {
        float a = i == at ? value : 0.f;
#pragma unroll 1
        for (uint32_t j = at; j < i; ++j) a -= F[i * ld + j] * y[j];
        y[i] = a;
        r += a * a / F[i * ld + i];
    }
    return r;
}

// The same for dense rows (contact rows against the articulation), all lanes on one row at a time: lane = coordinate
// in the forward solve, then lane = row adds its row's terms in coordinate order, so the sum is the sequential one.
// Results land in HF_RHO of each head (a field init_heads fills afterwards).
template <int NR>
NKB_DEV void mass_coupling_dense(Env& e, const Tile& tile) {
    const TemplateView& t = *e.t;
    const uint32_t n = t.ndof, ld = e.lay->ld, l = e.lane;
    if (n == 0u) return;
    const float* F = sm_factor(e);
    float* terms = e.sm + e.lay->chol;                  // Newton scratch, free until the first descent: >= n x n words
    const uint32_t batch = n < 32u ? n : 32u;           // rows per batch
    float diag[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) { const uint32_t c = l + 32u * r; diag[r] = c < n ? F[c * ld + c] : 1.f; }
#pragma unroll 1
    for (uint32_t base = 0u; base < tile.nheads; base += 32u) {
        const uint32_t h = base + l;
        bool dense = false;
        if (h < tile.nheads) {
            const uint32_t o = hu(e, HF_OWNER, h);
            dense = ((o & 0xffffu) == t.B || (o >> 16) == t.B) && !(hu(e, HF_JOFF, h) & kUnitRow);
        }
        uint32_t todo = __ballot_sync(NKB_FULL, dense);
#pragma unroll 1
        while (todo != 0u) {
            uint32_t in_batch = 0u, mine = 0xffffffffu;
#pragma unroll 1
            for (; todo != 0u && in_batch < batch; ++in_batch) {
                const uint32_t src = (uint32_t)__ffs(todo) - 1u;
                todo &= todo - 1u;
                if (l == src) mine = in_batch;
                const float* row = sm_jpool(e) + hu(e, HF_JOFF, base + src);
                float x[NR];
#pragma unroll
                for (int r = 0; r < NR; ++r) { const uint32_t c = l + 32u * r; x[r] = c < n ? row[c] : 0.f; }
#pragma unroll 1
                for (uint32_t j = 0u; j < n; ++j) {
                    const float xj = coord_bcast<NR>(x, j);
#pragma unroll
                    for (int r = 0; r < NR; ++r) { const uint32_t c = l + 32u * r; if (c > j && c < n) x[r] -= F[c * ld + j] * xj; }
                }
#pragma unroll
                for (int r = 0; r < NR; ++r) { const uint32_t c = l + 32u * r; if (c < n) terms[in_batch * n + c] = x[r] * x[r] / diag[r]; }
            }
            __syncwarp();
            if (mine != 0xffffffffu) {
                float r = 0.f;
#pragma unroll 1
                for (uint32_t i = 0u; i < n; ++i) r += terms[mine * n + i];
                hf(e, HF_RHO, h) = r;
            }
            __syncwarp();
        }
    }
}

// The same for contact rows between two branches of the tree, through a whole solve with the tree's factor.
template <int NR>
NKB_DEV void mass_coupling_branching(Env& e, const Tile& tile) {
    const TemplateView& t = *e.t;
#pragma unroll 1
    for (uint32_t h = 0u; h < tile.nheads; ++h) {
        const uint32_t o = hu(e, HF_OWNER, h), jo = hu(e, HF_JOFF, h);
        if (((o & 0xffffu) != t.B && (o >> 16) != t.B) || (jo & kUnitRow)) continue;
        const float* row = sm_jpool(e) + jo;
        float g[NR], x[NR], sum = 0.f;
#pragma unroll
        for (int r = 0; r < NR; ++r) g[r] = e.lane + 32u * r < t.ndof ? row[e.lane + 32u * r] : 0.f;
        solve_block_mass<NR>(e, t.B, g, x);
#pragma unroll
        for (int r = 0; r < NR; ++r) sum = fmaf(g[r], x[r], sum);
        sum = warp_sum(sum);
        if (e.lane == 0u) hf(e, HF_RHO, h) = sum;
        __syncwarp();
    }
}

// A contact between two branches of the tree couples all joints on both.  Eliminating the joints from the largest coordinate to the
// smallest (children before parents) then fills in just what the elimination tree of the coupled matrix says (Liu, The role of
// elimination trees in sparse factorization, SIAM J. Matrix Anal. Appl. 11, 1990): the parent of a joint is the largest coordinate
// left in its column, and the rest of the column passes on to the parent.  Two legs become one chain of twelve, an arm and a leg
// one of sixteen with the waist between them, and the solve goes on as on any tree.  Leaves the lanes' table in shared memory; returns the
// depth, 0 where it exceeds the levels the solve holds.  (4 steps of 2048 humanoids: 7.2 ms with dense systems
// where two limbs touch, 4.0 so; of 20 2.42 and 1.51.)
template <int NR>
NKB_DEV uint32_t merge_trees(Env& e, uint32_t nheads) {
    constexpr int kLevels = kSolveLevels<NR>;
    const TemplateView& t = *e.t;
    const uint32_t l = e.lane, n = t.ndof, n4 = (n + 3u) & ~3u, first = t.floating_root ? 6u : 0u, words = merged_lane_words(n);
    const TreeLane<kTreeLevels> tl = tree_lane(e);
    const bool joint = tl.level != kTreeNone;
    const uint32_t high = NR > 1 && n > 32u ? (1u << (n - 32u)) - 1u : 0u;        // lanes whose joint is one of the coordinates from 32 on
    const auto largest = [&](uint32_t lanes) { return 31u - (uint32_t)__clz((lanes & high) != 0u ? lanes & high : lanes); };
    const auto below = [&](uint32_t c) { return c < 32u ? ~high & ((1u << c) - 1u) : ~high | ((1u << (c - 32u)) - 1u); };        // lanes of smaller coordinates
    uint32_t column = 0u, desc = 0u;                 // lanes left in this joint's column, its descendants
#pragma unroll
    for (int p = 0; p < kTreeLevels; ++p) if (joint && (uint32_t)p < tl.level) column |= 1u << (tl.ancestor(p) & 31u);
#pragma unroll 1
    for (uint32_t h = 0u; h < nheads; ++h) {
        const uint32_t jo = hu(e, HF_JOFF, h);
        if (jo & kUnitRow) break;                    // contact heads come first
        const uint32_t owner = hu(e, HF_OWNER, h);
        if ((owner & 0xffffu) != t.B && (owner >> 16) != t.B) continue;
        const float* row = sm_jpool(e) + jo + tl.coord;
        const uint32_t acts = __ballot_sync(NKB_FULL, joint && (row[0] != 0.f || row[n4] != 0.f || row[2u * n4] != 0.f));
        if (joint && ((acts >> l) & 1u)) column |= acts & below(tl.coord);
    }
    uint32_t parent = 32u;
#pragma unroll 1
    for (uint32_t c = n; c > first; --c) {
        const uint32_t lane = (c - 1u) & 31u, left = __shfl_sync(NKB_FULL, column, lane), under = __shfl_sync(NKB_FULL, desc, lane);
        const uint32_t up = left != 0u ? largest(left) : 32u;
        if (l == lane) parent = up;
        if (l == up) { column |= left & ~(1u << l); desc |= under | (1u << lane); }
    }
    // the path to the root: the parent's path and the parent
    uint32_t* table = reinterpret_cast<uint32_t*>(e.sm + e.lay->merged);
    uint32_t* mine = table + l * words;
    if (!joint) { mine[0] = tl.coord | (kTreeNone << 8); mine[1] = 0u; for (uint32_t k = 2u; k < words; ++k) mine[k] = 0u; }
    uint32_t depth = 0u;
    __syncwarp();
#pragma unroll 1
    for (uint32_t c = first; c < n; ++c) {
        if (l == (c & 31u) && joint) {
            uint32_t level = 0u;
            for (uint32_t k = 2u; k < words; ++k) mine[k] = parent < 32u ? table[parent * words + k] : 0u;
            if (parent < 32u) {
                const uint32_t head = table[parent * words];
                level = ((head >> 8) & 0xffu) + 1u;
                if (level <= (uint32_t)kLevels) reinterpret_cast<uint8_t*>(mine + 2u)[level - 1u] = (uint8_t)(head & 0xffu);
            }
            mine[0] = tl.coord | (min(level, 0xfeu) << 8); mine[1] = desc;
            depth = level + 1u;
        }
        __syncwarp();
    }
    depth = __reduce_max_sync(NKB_FULL, depth);
    return depth <= (uint32_t)kLevels ? depth : 0u;
}

// Head setup: penalty, response scales (block_descent_tile.cuh:743-797).
template <int NR, bool kRows>
NKB_DEV void init_heads(Env& e, const Tile& tile, bool by_rows) {
    const TemplateView& t = *e.t;
    if (tile.nheads == 0u && !by_rows) return;
    if constexpr (NR > 0) {
        bool built = false;
        if constexpr (kRows) { if (by_rows && t.row_cap != 0u) built = build_rows<NR>(e, tile.nheads); }
        if (built) e.by_rows = kRowsFresh;
        else if (t.mass_tree == 0u) mass_coupling_dense<NR>(e, tile);
        else if (e.branching) mass_coupling_branching<NR>(e, tile);
    }
#pragma unroll 1
    for (uint32_t h = e.lane; h < tile.nheads; h += 32u) {
        float shares[2] = {0.f, 0.f};
        const uint32_t fl = hu(e, HF_FLAGS, h);
        const uint32_t jo = hu(e, HF_JOFF, h);
        bool valid = true;
#pragma unroll 1
        for (uint32_t side = 0u; side < 2u; ++side) {
            const uint32_t ob = head_owner(e, h, side);
            float c = 0.f;
            if (ob == kNoBlock16) { /* static or kinematic side: no response */ }
            else if (ob == t.B) {
                if constexpr (NR > 0) {
                    const bool unit = (jo & kUnitRow) != 0u;
                    if (kRows && e.by_rows != 0u) c = hf(e, HF_RHO, h);
                    else if (t.mass_tree != 0u && (unit || !e.branching))
                        c = tree_coupling<NR>(e, sm_factor(e), unit ? nullptr : sm_jpool(e) + jo, unit ? jo & 0xffffu : hu(e, HF_RHO, h), hf(e, HF_UNITV, h));
                    else if (unit) c = mass_coupling_unit<NR>(e, jo & 0xffffu, hf(e, HF_UNITV, h));
                    else c = hf(e, HF_RHO, h);
                }
            } else {
                const V3 dir = hf3(e, HF_N, h) * (side == 0u ? 1.f : -1.f);
                const V3 ang = cross(hf3(e, side == 0u ? HF_RA : HF_RB, h), dir);
                c = __ldg(t.inv_mass + ob) * dot(dir, dir) + dot(ang, sym_mulv(sm_bwinv(e, ob), ang));
            }
            valid &= c >= 0.f && isfinite(c);
            shares[side] = c;
        }
        const float response = (valid && isfinite(shares[0] + shares[1])) ? shares[0] + shares[1] : nanf("");
        const float coupling = shares[0] * shares[1], largest = fmaxf(shares[0], shares[1]);
        const float coupled = coupling > 0.f ? (response + sqrtf(response * response + 12.0f * coupling)) / (6.0f * coupling) : FLT_MAX;
        const float cap = 100.0f / largest;
        float rho = response > 0.f ? fminf(cap, coupled) : 0.f;
        if (!(response == 0.f || (response > 0.f && rho > 0.f && rho <= FLT_MAX))) { e.status |= kStatusSolverFailure; rho = nanf(""); }
        hf(e, HF_RHO, h) = rho;
        hst3(e, HF_BASE, h, hf3(e, HF_DUAL, h));
        hst3(e, HF_RES, h, mk3(0.f, 0.f, 0.f)); hst3(e, HF_MOVE, h, mk3(0.f, 0.f, 0.f)); hst3(e, HF_STEP, h, mk3(0.f, 0.f, 0.f));
        hst3(e, HF_RXS, h, mk3(0.f, 0.f, 0.f)); hf(e, HF_RXW, h) = 0.f; hst3(e, HF_RXP, h, mk3(0.f, 0.f, 0.f));
        (void)fl;
    }
    __syncwarp();
    if constexpr (kRows) {
        if (e.by_rows != 0u) {
            bool stiff = false;
            if (e.lane < e.rows) stiff = !(hf(e, HF_RHO, row_table(e)[e.lane] & 0xffffu) * row_w(e)[e.lane * (row_words(e) + 1u)] <= kRowStiffness);
            if (__any_sync(NKB_FULL, stiff)) e.by_rows = kRowsNone;
        }
    }
}

// Incidence lists (heads of each block in head order) and greedy colours.  Without free bodies the articulation is the only block; one
// of fixed joints alone is none, and rows that act on no block (a fixed link on the ground) are left as they are.
template <bool kRigid>
NKB_DEV void index_blocks(Env& e, Tile& tile, bool color) {
    const uint32_t nb = tile.nblocks;
    if (!kRigid && tile.nheads == 0u) {                 // the articulation alone, no row on it
        if (e.lane == 0u) {
            if (nb != e.t->B) blk_inc_begin(e, nb, e.t->B) = 0u;
            blk_inc_begin(e, nb, nb) = 0u;
            block_order(e, nb)[0] = e.t->B; block_order(e, nb)[nb] = nb - e.t->B;
        }
        tile.units = false;
        __syncwarp();
        return;
    }
    uint32_t* inc = blk_inc(e, nb);
    uint32_t at = 0u;
#pragma unroll 1
    for (uint32_t b = kRigid ? 0u : e.t->B; b < nb; ++b) {
        if (e.lane == 0u) blk_inc_begin(e, nb, b) = at;
        if (kRigid && blk_dim(e, b) == 0u) continue;                // no row acts on a block that does not move
#pragma unroll 1
        for (uint32_t base = 0u; base < tile.nheads; base += 32u) {
            const uint32_t h = base + e.lane;
            bool hit = false;
            if (h < tile.nheads) { const uint32_t o = hu(e, HF_OWNER, h); hit = (o & 0xffffu) == b || (o >> 16) == b; }
            const uint32_t m = __ballot_sync(NKB_FULL, hit);
            if (hit) inc[at + __popc(m & ((1u << e.lane) - 1u))] = h;
            at += __popc(m);
        }
    }
    if (e.lane == 0u) blk_inc_begin(e, nb, nb) = at;
    __syncwarp();
    // contact heads come first in an incidence list, rows on a single coordinate last
    tile.units = at != 0u && (hu(e, HF_JOFF, inc[at - 1u]) & kUnitRow) != 0u && ((hu(e, HF_OWNER, inc[at - 1u]) & 0xffffu) == e.t->B);
    if (tile.units) {
        uint16_t* utab = unit_table(e, nb);
#pragma unroll 1
        for (uint32_t k = e.lane; k < 3u * e.vstride; k += 32u) utab[k] = (uint16_t)kNoUnitHead;
        __syncwarp();
#pragma unroll 1
        for (uint32_t h = e.lane; h < tile.nheads; h += 32u) {
            const uint32_t jo = hu(e, HF_JOFF, h), o = hu(e, HF_OWNER, h), fl = hu(e, HF_FLAGS, h);
            if (!(jo & kUnitRow) || ((o & 0xffffu) != e.t->B && (o >> 16) != e.t->B)) continue;
            const uint32_t slot = (fl & kHeadFriction) ? 2u : hf(e, HF_UNITV, h) < 0.f ? 1u : 0u;
            utab[slot * e.vstride + (jo & 0xffffu)] = (uint16_t)h;
        }
        __syncwarp();
    }
    if constexpr (!kRigid) {
        if (color && e.lane == 0u) { block_order(e, nb)[0] = e.t->B; block_order(e, nb)[nb] = nb - e.t->B; }
        __syncwarp();
        return;
    }
    if (!color) return;
    uint32_t colours = 0u;       // 1 + the largest colour in use
#pragma unroll 1
    for (uint32_t b = 0u; b < nb; ++b) {
        if (blk_dim(e, b) == 0u) { if (e.lane == 0u) blk_color(e, nb, b) = 0xffffffffu; continue; }
        uint32_t taken = 0u;
        const uint32_t ib = blk_inc_begin(e, nb, b), ie = blk_inc_begin(e, nb, b + 1u);
#pragma unroll 1
        for (uint32_t k = ib + e.lane; k < ie; k += 32u) {
            const uint32_t o = hu(e, HF_OWNER, inc[k]);
            const uint32_t first = o & 0xffffu, second = o >> 16;
            const uint32_t other = first == b ? second : first;
            if (other < b && blk_dim(e, other) != 0u) taken |= 1u << blk_color(e, nb, other);
        }
        taken = __reduce_or_sync(NKB_FULL, taken);
        const uint32_t c = min((uint32_t)__ffs(~taken) - 1u, 31u);
        colours = max(colours, c + 1u);
        if (e.lane == 0u) blk_color(e, nb, b) = c;
        __syncwarp();
    }
    __syncwarp();
    // descent order: colour by colour, index order inside a colour (block_descent_tile.cuh:2749-2820)
    uint32_t* order = block_order(e, nb);
    uint32_t count = 0u;
#pragma unroll 1
    for (uint32_t c = 0u; c < colours; ++c)
#pragma unroll 1
        for (uint32_t base = 0u; base < nb; base += 32u) {
            const uint32_t b = base + e.lane;
            const bool hit = b < nb && blk_color(e, nb, b) == c;
            const uint32_t m = __ballot_sync(NKB_FULL, hit);
            if (hit) order[count + __popc(m & ((1u << e.lane) - 1u))] = b;
            count += __popc(m);
        }
    if (e.lane == 0u) order[nb] = count;
    __syncwarp();
}

// residual = rhs dt - J u at the blocks' current velocities (block_descent_tile.cuh:891-930); lane = axis of a head
NKB_DEV void init_residuals(Env& e, const Tile& tile) {
    const TemplateView& t = *e.t;
    const float dt = t.cfg.dt;
#pragma unroll 1
    for (uint32_t k = e.lane; k < 3u * tile.nheads; k += 32u) {
        const uint32_t h = k / 3u, ax = k - 3u * h;
        float along = 0.f;
        const bool live = ax < head_axes(e, h);
        if (live)
#pragma unroll 1
            for (uint32_t side = 0u; side < 2u; ++side) {
                const uint32_t b = head_owner(e, h, side);
                if (b == kNoBlock16) continue;
                along += head_row_dot(e, h, side, ax, b, block_vel(e, b, false));
            }
        hf(e, HF_RES + ax, h) = live ? (ax == 0u ? hf(e, HF_RHS, h) * dt : 0.f) - along : 0.f;
    }
    __syncwarp();
}

// Leading dimension of a shared-memory matrix whose rows are read as float4 by one lane per row:
// a multiple of 4 words that is 4 mod 8, so the eight lanes of a quarter warp hit distinct bank groups.
NKB_DEV uint32_t pad_ld(uint32_t n) { const uint32_t ld = (n + 3u) & ~3u; return (ld & 7u) == 0u ? ld + 4u : ld; }

// Register copy of one head for the row evaluations.
struct HeadRegs {
    V3 dual, res, move, step;
    float rho, lower, upper, mu;
    bool cone;      // contact head with friction (the position pass clears the coefficient of its scalar rows)
};
NKB_DEV HeadRegs load_head(const Env& e, uint32_t h) {
    HeadRegs r;
    const float4 dual = hq(e, HF_DUAL, h), res = hq(e, HF_RES, h), move = hq(e, HF_MOVE, h), step = hq(e, HF_STEP, h);
    r.dual = mk3(dual.x, dual.y, dual.z); r.res = mk3(res.x, res.y, res.z);
    r.move = mk3(move.x, move.y, move.z); r.step = mk3(step.x, step.y, step.z);
    r.rho = dual.w; r.mu = res.w; r.lower = move.w; r.upper = step.w;
    r.cone = r.mu > 0.f;
    return r;
}
// The friction cone's radius follows the head's normal multiplier at the start of the descent, which the descent leaves as it is.
NKB_DEV void respond(const HeadRegs& r, V3 move, V3& f, float& cxx, float& cyy, float& czz, float& cyz) {
    const STerm n = scalar_impulse(r.dual.x, r.rho, r.res.x - move.x, r.lower, r.upper);
    f = mk3(n.impulse, 0.f, 0.f);
    cxx = n.curvature; cyy = czz = cyz = 0.f;
    if (r.cone) cone_impulse(r.dual, r.rho, r.res.y - move.y, r.res.z - move.z, r.dual.x, r.mu, f.y, f.z, cyy, czz, cyz);
}

// Row steps J d of the articulation's incident heads (block_descent_tile.cuh:2019-2044); lane = axis of a head, d staged in shared
// memory with zeros past the block's dimension.
NKB_DEV void row_steps(Env& e, const uint32_t* inc, uint32_t ib, uint32_t ie, uint32_t dim, const float* dvec) {
    const uint32_t chunks = (dim + 3u) >> 2;
    const float4* d4 = reinterpret_cast<const float4*>(dvec);
#pragma unroll 1
    for (uint32_t k = e.lane; k < 3u * (ie - ib); k += 32u) {
        const uint32_t at = k / 3u, ax = k - 3u * at, h = inc[ib + at];
        const uint32_t jo = hu(e, HF_JOFF, h);
        float s = 0.f;
        if (ax < head_axes(e, h)) {
            if (jo & kUnitRow) s = hf(e, HF_UNITV, h) * dvec[jo & 0xffffu];
            else {
                const float4* j4 = reinterpret_cast<const float4*>(sm_jpool(e) + jo) + ax * chunks;
#pragma unroll 1
                for (uint32_t c = 0u; c < chunks; ++c) {
                    const float4 d = d4[c], r = j4[c];
                    s = fmaf(r.x, d.x, s); s = fmaf(r.y, d.y, s); s = fmaf(r.z, d.z, s); s = fmaf(r.w, d.w, s);
                }
            }
        }
        hf(e, HF_STEP + ax, h) = s;
    }
    __syncwarp();
}

// One head's share of the line derivatives at step length alpha.
NKB_DEV void line_terms(const HeadRegs& r, float alpha, CSum& rs, float& rc, float& rm) {
    const V3 trial = mk3(fmaf(alpha, r.step.x, r.move.x), fmaf(alpha, r.step.y, r.move.y), fmaf(alpha, r.step.z, r.move.z));
    V3 f; float cxx, cyy, czz, cyz;
    respond(r, trial, f, cxx, cyy, czz, cyz);
    csum_addp(rs, f.x, r.step.x); csum_addp(rs, f.y, r.step.y); csum_addp(rs, f.z, r.step.z);
    rm += (fabsf(f.x) + kImpulseRounding * cxx * (fabsf(r.res.x) + fabsf(trial.x))) * fabsf(r.step.x) +
          (fabsf(f.y) + kImpulseRounding * cyy * (fabsf(r.res.y) + fabsf(trial.y))) * fabsf(r.step.y) +
          (fabsf(f.z) + kImpulseRounding * czz * (fabsf(r.res.z) + fabsf(trial.z))) * fabsf(r.step.z);
    rc += cxx * r.step.x * r.step.x + cyy * r.step.y * r.step.y + czz * r.step.z * r.step.z + 2.0f * cyz * r.step.y * r.step.z;
}

// Exact line search on the block's one-dimensional model (block_descent_tile.cuh:2048-2125): the first
// evaluation (alpha = 0) gives the initial slope, the following ones bracket and polish the root.  With at most
// 32 incident heads each lane keeps its head in registers for the whole search.  `fixed` is this lane's share of the constant impulses'
// slope, unrounded like the rows' slopes.
NKB_DEV float search_line(Env& e, const Tile& tile, uint32_t b, float islope, float icurv, const CSum& fixed, float fixed_size) {
    const uint32_t nb = tile.nblocks;
    const uint32_t* inc = blk_inc(e, nb);
    const uint32_t ib = blk_inc_begin(e, nb, b), ie = blk_inc_begin(e, nb, b + 1u);
    const bool single = ie - ib <= 32u, mine = ib + e.lane < ie;
    HeadRegs cached;
    if (single && mine) cached = load_head(e, inc[ib + e.lane]);
    float low = 0.0f, high = 0.0f, alpha = 0.0f, initial = 0.0f, result = 0.0f;
    bool bounded = false, have = false;
#pragma unroll 1
    for (int step = -1; step < (int)kLineSteps; ++step) {
        CSum rs = {0.f, 0.f};
        float rc = 0.f, rm = 0.f;
        if (single) { if (mine) line_terms(cached, alpha, rs, rc, rm); }
        else
#pragma unroll 1
        for (uint32_t k = ib + e.lane; k < ie; k += 32u) { const HeadRegs r = load_head(e, inc[k]); line_terms(r, alpha, rs, rc, rm); }
        CSum total = {-rs.value, -rs.error};
        csum_add(total, -fixed.value); csum_add(total, -fixed.error);
        if (e.lane == 0u) { csum_addp(total, alpha, icurv); csum_add(total, islope); }
        const float slope = warp_csum_total(total);
        const float curvature = icurv + warp_sum(rc);
        const float magnitude = fabsf(islope) + alpha * icurv + fixed_size + warp_sum(rm);
        if (step < 0) {
            initial = slope;
            if (!(initial < 0.0f)) { have = true; result = 0.0f; break; }
            alpha = 1.0f;
            continue;
        }
        if (!isfinite(slope) || !isfinite(curvature)) { high = alpha; bounded = true; alpha = 0.5f * (low + high); continue; }
        if (fabsf(slope) <= fmaxf(kLineTol * -initial, kRoundings * FLT_EPSILON * magnitude)) { have = true; result = alpha; break; }
        if (slope < 0.0f) low = alpha; else { high = alpha; bounded = true; }
        if (bounded && high - low <= FLT_EPSILON * high) break;
        float next = alpha - __fdividef(slope, curvature);
        if (!(next > low && (!bounded || next < high))) next = bounded ? 0.5f * (low + high) : 2.0f * alpha;
        alpha = next;
    }
    return have ? result : low;
}

NKB_DEV void apply_moves(Env& e, const Tile& tile, uint32_t b, float alpha) {
    const uint32_t nb = tile.nblocks;
    const uint32_t* inc = blk_inc(e, nb);
    const uint32_t ib = blk_inc_begin(e, nb, b), ie = blk_inc_begin(e, nb, b + 1u);
#pragma unroll 1
    for (uint32_t k = ib + e.lane; k < ie; k += 32u) {
        const uint32_t h = inc[k];
        const V3 step = hf3(e, HF_STEP, h), move = hf3(e, HF_MOVE, h);
        hst3(e, HF_MOVE, h, mk3(fmaf(alpha, step.x, move.x), fmaf(alpha, step.y, move.y), fmaf(alpha, step.z, move.z)));
    }
    __syncwarp();
}

// A descent whose force is within its own rounding while M^-1 times that rounding stays above the tolerance (light links) goes on to the step limit,
// 1e-7 m/s a step.  Ending it there is no less exact against 64 bits and up to 1.3 times faster (rollouts of 2500 quadrupeds), but such steps move
// single envs across the edge of a contact: one batch of six was 3.5e-3 from the results with all steps, piles 0.3 in one box.  It is not done.
//
// Newton steps with exact line search on one block, from where it stands.  A descent ends at the block's minimum wherever it begins, to
// rounding, so the reference's search toward the free velocity ahead of the first sweep's Newton steps (block_descent_tile.cuh:2196-2210)
// is left out: with it a policy step of 1000 quadrupeds took 2 % more line evaluations and time, 4096 quadrupeds with 4 boxes 5 %.
// Where sweeps end at their limit, or a comparison picks a contact's axis, an env shows the other rounding amplified; against 64 bits
// both are as far off (linear velocities of 48-box piles after two steps: relative 1.71e-4 either way).  A lane owns coordinates lane + 32 r (r < NR) and the same rows of
// the Newton matrix, which lives in the env's shared-memory slice in float4-readable rows; lane k also owns the k-th
// incident head in the row evaluations and publishes its response through the head's shared-memory fields.
template <int NR>
NKB_DEV void descend_block(Env& e, Tile& tile, uint32_t b, bool position) {
    const uint32_t l = e.lane, nb = tile.nblocks, dim = blk_dim(e, b);
    const uint32_t* inc = blk_inc(e, nb);
    const uint32_t ib = blk_inc_begin(e, nb, b), ie = blk_inc_begin(e, nb, b + 1u);
    // A block without a push-out row keeps its zero position correction: its descent would minimise u^T M u from u = 0.
    // (In the velocity phase an unconstrained block still has to reach its free velocity.)
    if (position && ib == ie) return;
    const uint32_t chunks = (dim + 3u) >> 2, ldh = pad_ld(dim);
    float* velocity = block_vel(e, b, position);
    float* dvec = sm_vec(e, kVecD);
    float* hi_v = sm_vec(e, kVecS0);
    float* lo_v = sm_vec(e, kVecS1);
    float* u_v = sm_vec(e, kVecS2);
    float* H = e.sm + e.lay->chol;
    bool coord[NR];
    float* Hr[NR];
    const float* Mr[NR];                // this lane's rows of the block mass, zero past the block's dimension
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const uint32_t c = l + 32u * r;
        coord[r] = c < dim;
        Hr[r] = H + (coord[r] ? c : 0u) * ldh;
        Mr[r] = sm_mass(e) + (coord[r] ? c : 0u) * e.lay->ld;
    }
    bool coupled = false;
#pragma unroll 1
    for (uint32_t k = ib + l; k < ie; k += 32u) {
        const uint32_t h = inc[k];
        const uint32_t o = hu(e, HF_OWNER, h);
        coupled |= (o & 0xffffu) != kNoBlock16 && (o >> 16) != kNoBlock16;
        hst3(e, HF_MOVE, h, mk3(0.f, 0.f, 0.f));
    }
    coupled = __any_sync(NKB_FULL, coupled);
    __syncwarp();
    float start[NR], fr[NR], u[NR], fixed[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        fixed[r] = position || !coord[r] ? 0.f : sm_fixed(e)[l + 32u * r];
        start[r] = coord[r] ? velocity[l + 32u * r] : 0.f;
        fr[r] = (coord[r] && !position) ? block_free(e, b)[l + 32u * r] : 0.f;
        u[r] = start[r];
    }
    bool failure = false;
    float primal = FLT_MAX;
    tick(e, 15);
#pragma unroll 1
    for (int step = 0; step < (int)kNewtonSteps; ++step) {
        float d[NR], force[NR], inertia[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) { d[r] = 0.f; force[r] = 0.f; inertia[r] = 0.f; }
        {
            // ---- lane = head: responses at the current moves, published to shared memory ----
            uint32_t dense_any = 0u;
#pragma unroll 1
            for (uint32_t k = ib + l; k < ie; k += 32u) {
                const uint32_t h = inc[k];
                const HeadRegs hr = load_head(e, h);
                V3 f; float cxx, cyy, czz, cyz;
                respond(hr, hr.move, f, cxx, cyy, czz, cyz);
                const V3 noise = mk3(fabsf(f.x) + cxx * (fabsf(hr.res.x) + fabsf(hr.move.x)), fabsf(f.y) + cyy * (fabsf(hr.res.y) + fabsf(hr.move.y)),
                                     fabsf(f.z) + czz * (fabsf(hr.res.z) + fabsf(hr.move.z)));
                hst3(e, HF_F, h, f); hst3(e, HF_NZ, h, noise);
                hf(e, HF_C, h) = cxx; hf(e, HF_C + 1u, h) = cyy; hf(e, HF_C + 2u, h) = czz; hf(e, HF_C + 3u, h) = cyz;
                const bool contributes = f.x != 0.f || f.y != 0.f || f.z != 0.f || cxx != 0.f || cyy != 0.f || czz != 0.f || cyz != 0.f ||
                                         noise.x != 0.f || noise.y != 0.f || noise.z != 0.f;
                const bool unit = (hu(e, HF_JOFF, h) & kUnitRow) != 0u;
                dense_any |= (contributes && !unit) ? 1u : 0u;
            }
            // ---- lane = coordinate: inertial part of H (rows of this lane) and g ----
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const float diff = u[r] - fr[r];
                const float part = diff - u[r];
                const float diff_err = (u[r] - (diff - part)) + (-fr[r] - part);
                hi_v[l + 32u * r] = diff; lo_v[l + 32u * r] = diff_err; u_v[l + 32u * r] = u[r];
            }
            __syncwarp();
            CSum inertial[NR], g[NR];
            float scale[NR], diag[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                inertial[r].value = 0.f; inertial[r].error = 0.f;
                scale[r] = 0.f; diag[r] = 0.f;
                if (coord[r]) {
                    const float4* Mr4 = reinterpret_cast<const float4*>(Mr[r]);
                    float4* Hr4 = reinterpret_cast<float4*>(Hr[r]);
#pragma unroll 1
                    for (uint32_t c = 0u; c < chunks; ++c) {
                        const float4 m = Mr4[c], hi = reinterpret_cast<const float4*>(hi_v)[c], lo = reinterpret_cast<const float4*>(lo_v)[c];
                        Hr4[c] = m;
                        csum_addp(inertial[r], m.x, hi.x); inertial[r].error = fmaf(m.x, lo.x, inertial[r].error);
                        csum_addp(inertial[r], m.y, hi.y); inertial[r].error = fmaf(m.y, lo.y, inertial[r].error);
                        csum_addp(inertial[r], m.z, hi.z); inertial[r].error = fmaf(m.z, lo.z, inertial[r].error);
                        csum_addp(inertial[r], m.w, hi.w); inertial[r].error = fmaf(m.w, lo.w, inertial[r].error);
                        scale[r] += fabsf(m.x) * fabsf(hi.x) + fabsf(m.y) * fabsf(hi.y) + fabsf(m.z) * fabsf(hi.z) + fabsf(m.w) * fabsf(hi.w);
                    }
                }
                g[r].value = -inertial[r].value; g[r].error = -inertial[r].error;
            }
            tick(e, 16);
            // rows on a single coordinate only touch that coordinate (block_descent_tile.cuh:1555-1568)
            if (tile.units) {
                const uint16_t* utab = unit_table(e, nb);
                const uint32_t vs = e.vstride;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
#pragma unroll 1
                    for (uint32_t slot = 0u; slot < 3u; ++slot) {
                        const uint32_t h = utab[slot * vs + l + 32u * r];
                        if (h == kNoUnitHead) continue;
                        const float v = hf(e, HF_UNITV, h);
                        diag[r] += v * hf(e, HF_C, h) * v;
                        csum_addp(g[r], v, hf(e, HF_F, h));
                        scale[r] += fabsf(v) * hf(e, HF_NZ, h);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) { csum_add(g[r], fixed[r]); scale[r] += fabsf(fixed[r]); }
            // dense rows: H += J^T C J, g += J^T f, one head at a time with its values broadcast from shared memory
            if (__any_sync(NKB_FULL, dense_any != 0u)) {
#pragma unroll 1
                for (uint32_t k = ib; k < ie; ++k) {
                    const uint32_t hs = inc[k];
                    const uint32_t jo = hu(e, HF_JOFF, hs);
                    if (jo & kUnitRow) continue;
                    const V3 f = hf3(e, HF_F, hs), nz = mk3(hf(e, HF_NZ, hs), hf(e, HF_NZ + 1u, hs), hf(e, HF_NZ + 2u, hs));
                    const float c0 = hf(e, HF_C, hs), c1 = hf(e, HF_C + 1u, hs), c2 = hf(e, HF_C + 2u, hs), c12 = hf(e, HF_C + 3u, hs);
                    if (!(f.x != 0.f || f.y != 0.f || f.z != 0.f || c0 != 0.f || c1 != 0.f || c2 != 0.f || c12 != 0.f || nz.x != 0.f || nz.y != 0.f || nz.z != 0.f)) continue;
                    const float* jr = sm_jpool(e) + jo;
                    const uint32_t js = chunks << 2;
                    const float4* r0 = reinterpret_cast<const float4*>(jr);
                    const float4* r1 = reinterpret_cast<const float4*>(jr + js);
                    const float4* r2 = reinterpret_cast<const float4*>(jr + 2u * js);
#pragma unroll
                    for (int r = 0; r < NR; ++r) {
                        const uint32_t c = l + 32u * r;
                        const float j0 = coord[r] ? jr[c] : 0.f, j1 = coord[r] ? jr[js + c] : 0.f, j2 = coord[r] ? jr[2u * js + c] : 0.f;
                        csum_addp(g[r], j0, f.x); csum_addp(g[r], j1, f.y); csum_addp(g[r], j2, f.z);
                        scale[r] += fabsf(j0) * nz.x + fabsf(j1) * nz.y + fabsf(j2) * nz.z;
                        const float a0 = j0 * c0, a1 = j1 * c1 + j2 * c12, a2 = j2 * c2 + j1 * c12;
                        if (coord[r]) {
                            float4* Hr4 = reinterpret_cast<float4*>(Hr[r]);
#pragma unroll 1
                            for (uint32_t cc = 0u; cc < chunks; ++cc) {
                                float4 h4 = Hr4[cc];
                                const float4 x = r0[cc], y = r1[cc], z = r2[cc];
                                h4.x += a0 * x.x + a1 * y.x + a2 * z.x;
                                h4.y += a0 * x.y + a1 * y.y + a2 * z.y;
                                h4.z += a0 * x.z + a1 * y.z + a2 * z.z;
                                h4.w += a0 * x.w + a1 * y.w + a2 * z.w;
                                Hr4[cc] = h4;
                            }
                        }
                    }
                }
            }
            tick(e, 17);
            bool finite = true, small = true;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                if (coord[r]) {
                    float4* Hr4 = reinterpret_cast<float4*>(Hr[r]);
                    Hr[r][l + 32u * r] += diag[r];
#pragma unroll 1
                    for (uint32_t c = 0u; c < chunks; ++c) {
                        const float4 v = Hr4[c], uu = reinterpret_cast<const float4*>(u_v)[c];
                        finite &= isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w);
                        scale[r] += fabsf(v.x) * fabsf(uu.x) + fabsf(v.y) * fabsf(uu.y) + fabsf(v.z) * fabsf(uu.z) + fabsf(v.w) * fabsf(uu.w);
                    }
                    force[r] = g[r].value + g[r].error; inertia[r] = inertial[r].value + inertial[r].error;
                }
                finite &= isfinite(force[r]);
                small &= !coord[r] || fabsf(force[r]) <= kRoundings * FLT_EPSILON * scale[r];
            }
            if (!__all_sync(NKB_FULL, finite)) { failure = true; break; }
            bool converged = __all_sync(NKB_FULL, small);
            if (converged && tile.tol > 0.f) {
                solve_block_mass<NR>(e, b, force, d);
                bool still = true;
#pragma unroll
                for (int r = 0; r < NR; ++r) still &= !coord[r] || fabsf(d[r]) < tile.tol;
                converged = __all_sync(NKB_FULL, still);
            }
            if (converged) { primal = 0.f; break; }
            tick(e, 18);
            // ---- Cholesky, rows of L over the rows of H (block_descent_tile.cuh:1623-1641) ----
            bool valid = true;
            float inverse[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) inverse[r] = 0.f;
            __syncwarp();
#pragma unroll 1
            for (uint32_t k = 0u; k < dim; ++k) {
                float value[NR];
                const float4* Hk4 = reinterpret_cast<const float4*>(H + k * ldh);
                const uint32_t full = k >> 2, rem = k & 3u;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    value[r] = 0.f;
                    if (coord[r] && l + 32u * r >= k) {
                        const float4* Hr4 = reinterpret_cast<const float4*>(Hr[r]);
                        float s0 = 0.f, s1 = 0.f;
#pragma unroll 1
                        for (uint32_t c = 0u; c < full; ++c) {
                            const float4 a = Hr4[c], bb = Hk4[c];
                            s0 = fmaf(a.x, bb.x, s0); s1 = fmaf(a.y, bb.y, s1); s0 = fmaf(a.z, bb.z, s0); s1 = fmaf(a.w, bb.w, s1);
                        }
                        const float4 a = Hr4[full], bb = Hk4[full];
                        if (rem > 0u) s0 = fmaf(a.x, bb.x, s0);
                        if (rem > 1u) s1 = fmaf(a.y, bb.y, s1);
                        if (rem > 2u) s0 = fmaf(a.z, bb.z, s0);
                        value[r] = Hr[r][k] - (s0 + s1);
                    }
                }
                const float pivot = coord_bcast<NR>(value, k);
                valid &= pivot > 0.f && pivot <= FLT_MAX;
                const float sc = rsqrtf(valid ? pivot : 1.0f), root = pivot * sc;
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const uint32_t c = l + 32u * r;
                    if (coord[r] && c >= k) Hr[r][k] = c == k ? root : value[r] * sc;
                    inverse[r] = c == k ? sc : inverse[r];
                }
                __syncwarp();
            }
            if (!valid) { failure = true; break; }
            tick(e, 19);
            // ---- d = H^-1 g ----
            float rr[NR], scaled[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) rr[r] = force[r];
#pragma unroll 1
            for (uint32_t j = 0u; j < dim; ++j) {
#pragma unroll
                for (int r = 0; r < NR; ++r) scaled[r] = rr[r] * inverse[r];
                const float y = coord_bcast<NR>(scaled, j);
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const uint32_t c = l + 32u * r;
                    rr[r] = c == j ? y : ((coord[r] && c > j) ? fmaf(-Hr[r][j], y, rr[r]) : rr[r]);
                }
            }
#pragma unroll 1
            for (uint32_t jj = dim; jj > 0u; --jj) {
                const uint32_t j = jj - 1u;
#pragma unroll
                for (int r = 0; r < NR; ++r) scaled[r] = rr[r] * inverse[r];
                const float x = coord_bcast<NR>(scaled, j);
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const uint32_t c = l + 32u * r;
                    rr[r] = c == j ? x : (c < j ? fmaf(-H[j * ldh + c], x, rr[r]) : rr[r]);
                }
            }
#pragma unroll
            for (int r = 0; r < NR; ++r) d[r] = coord[r] ? rr[r] : 0.f;
        }
        // ---- curvature and slopes along d ----
        __syncwarp();
#pragma unroll
        for (int r = 0; r < NR; ++r) dvec[l + 32u * r] = d[r];
        __syncwarp();
        CSum dec = {0.f, 0.f}, slo = {0.f, 0.f}, cur = {0.f, 0.f}, fix = {0.f, 0.f};
        float fix_size = 0.f;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            float ms = 0.f;
            if (coord[r]) {
                const float4* Mr4 = reinterpret_cast<const float4*>(Mr[r]);
#pragma unroll 1
                for (uint32_t c = 0u; c < chunks; ++c) {
                    const float4 m = Mr4[c], dd = reinterpret_cast<const float4*>(dvec)[c];
                    ms = fmaf(m.x, dd.x, ms); ms = fmaf(m.y, dd.y, ms); ms = fmaf(m.z, dd.z, ms); ms = fmaf(m.w, dd.w, ms);
                }
                csum_addp(dec, force[r], d[r]); csum_addp(slo, inertia[r], d[r]); csum_addp(cur, d[r], ms); csum_addp(fix, fixed[r], d[r]); fix_size += fabsf(fixed[r] * d[r]);
            }
        }
        const float icurv = warp_csum_total(cur);
        const float total_dec = warp_csum_total(dec), islope = warp_csum_total(slo);
        if (!isfinite(total_dec) || !isfinite(islope) || !isfinite(icurv)) { failure = true; break; }
        if (!(total_dec > 0.f)) break;
        tick(e, 20);
        row_steps(e, inc, ib, ie, dim, dvec);
        tick(e, 21);
        const float alpha = search_line(e, tile, b, islope, icurv, fix, warp_sum(fix_size));
        tick(e, 22);
        tick_count(e, 23);
        float after[NR];
        bool fin_l = true, rounded_l = true;
        float step_l = 0.f;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            after[r] = fmaf(alpha, d[r], u[r]);
            fin_l &= !coord[r] || isfinite(after[r]);
            rounded_l &= !coord[r] || after[r] == u[r];
            step_l = fmaxf(step_l, coord[r] ? fabsf(alpha * d[r]) : 0.f);
        }
        const bool fin = __all_sync(NKB_FULL, fin_l);
        const bool rounded = __all_sync(NKB_FULL, rounded_l);
        if (!fin) { failure = true; break; }
        primal = warp_max(rounded ? 0.f : step_l);
        if (!(alpha > 0.f)) break;
#pragma unroll
        for (int r = 0; r < NR; ++r) u[r] = after[r];
        apply_moves(e, tile, b, alpha);
        if (rounded) break;
    }
#pragma unroll 1
    for (uint32_t k = ib + l; k < ie; k += 32u) {
        const uint32_t h = inc[k];
        const V3 res = hf3(e, HF_RES, h), move = hf3(e, HF_MOVE, h);
        hst3(e, HF_RES, h, mk3(__fsub_rn(res.x, move.x), __fsub_rn(res.y, move.y), __fsub_rn(res.z, move.z)));
    }
    if (failure) e.status |= kStatusSolverFailure;
    float moved = failure ? FLT_MAX : 0.f;
#pragma unroll
    for (int r = 0; r < NR; ++r) if (coord[r]) moved = fmaxf(moved, residual_abs(u[r] - start[r]));
    moved = warp_max(moved);
    tile.momentum = fmaxf(tile.momentum, moved);
    if (failure) primal = FLT_MAX;
    tile.residual = fmaxf(tile.residual, fmaxf(primal, coupled ? moved : 0.f));
#pragma unroll
    for (int r = 0; r < NR; ++r) if (coord[r]) velocity[l + 32u * r] = u[r];
    __syncwarp();
}

// One constraint row's share of an evaluation at step length alpha: adds to the line's slope, curvature and rounding magnitude,
// and leaves the head's impulse, curvature and noise scale at the trial point in its record, where the assembly of the next
// Newton system finds them.
NKB_DEV void evaluate_head(const Env& e, uint32_t h, float alpha, double& slope, float& curvature, float& magnitude) {
    const float4 dual = hq(e, HF_DUAL, h), res = hq(e, HF_RES, h), move = hq(e, HF_MOVE, h), step = hq(e, HF_STEP, h);
    const float rho = dual.w, lower = move.w, upper = step.w;
    const V3 trial = mk3(fmaf(alpha, step.x, move.x), fmaf(alpha, step.y, move.y), fmaf(alpha, step.z, move.z));
    const STerm n = scalar_impulse(dual.x, rho, res.x - trial.x, lower, upper);
    V3 f = mk3(n.impulse, 0.f, 0.f), noise = mk3(fmaf(n.curvature, fabsf(res.x) + fabsf(trial.x), fabsf(n.impulse)), 0.f, 0.f);
    float cyy = 0.f, czz = 0.f, cyz = 0.f;
    slope = fma((double)f.x, (double)step.x, slope);
    curvature = fmaf(n.curvature * step.x, step.x, curvature);
    magnitude = fmaf(fmaf(kImpulseRounding, noise.x - fabsf(f.x), fabsf(f.x)), fabsf(step.x), magnitude);
    if (res.w > 0.f) {
        cone_impulse(mk3(dual.x, dual.y, dual.z), rho, res.y - trial.y, res.z - trial.z, dual.x, res.w, f.y, f.z, cyy, czz, cyz);
        noise.y = fmaf(cyy, fabsf(res.y) + fabsf(trial.y), fabsf(f.y));
        noise.z = fmaf(czz, fabsf(res.z) + fabsf(trial.z), fabsf(f.z));
        slope = fma((double)f.y, (double)step.y, slope); slope = fma((double)f.z, (double)step.z, slope);
        curvature = fmaf(fmaf(cyy, step.y, cyz * step.z), step.y, fmaf(fmaf(czz, step.z, cyz * step.y), step.z, curvature));
        magnitude = fmaf(fmaf(kImpulseRounding, noise.y - fabsf(f.y), fabsf(f.y)), fabsf(step.y), magnitude);
        magnitude = fmaf(fmaf(kImpulseRounding, noise.z - fabsf(f.z), fabsf(f.z)), fabsf(step.z), magnitude);
    }
    hq(e, HF_F, h) = make_float4(f.x, f.y, f.z, n.curvature);
    hq(e, HF_C + 1u, h) = make_float4(cyy, czz, cyz, noise.x);
    *reinterpret_cast<float2*>(&hf(e, HF_NZ + 1u, h)) = make_float2(noise.y, noise.z);
}
// The rows of a block, lane = head, as many passes as the block has heads; 2 * half lanes take part.
NKB_DEV void evaluate_line(const Env& e, const uint32_t* inc, uint32_t ib, uint32_t ie, uint32_t half, float alpha, double& slope, float& curvature, float& magnitude) {
    slope = 0.0; curvature = 0.f; magnitude = 0.f;
#pragma unroll 1
    for (uint32_t k = ib + e.lane; k < ie; k += 32u) evaluate_head(e, inc[k], alpha, slope, curvature, magnitude);
    line_sums(slope, curvature, magnitude, half, e.lane);
}

// Row c of the mass matrix times a vector in shared memory (zeros past the last coordinate), in 64 bits.
NKB_DEV double mass_row_times(const Env& e, uint32_t c, uint32_t chunks, const double* v) {
    const float4* m4 = reinterpret_cast<const float4*>(sm_mass(e) + c * e.lay->ld);
    const double2* v2 = reinterpret_cast<const double2*>(v);
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 1
    for (uint32_t k = 0u; k < chunks; ++k) {
        const float4 m = m4[k];
        const double2 a = v2[2u * k], z = v2[2u * k + 1u];
        s0 = fma((double)m.x, a.x, s0); s1 = fma((double)m.y, a.y, s1); s0 = fma((double)m.z, z.x, s0); s1 = fma((double)m.w, z.y, s1);
    }
    return s0 + s1;
}

// The articulation's descent with the Newton system kept in the sparsity of its tree (nkb_tree.cuh).  Same model, stopping
// rules and exact line search as descend_block; contact rows act along root paths of the tree, or of the one merge_trees made.
//
// What bounds it is instruction supply: an SM keeps 32 KB of instructions close and fetches the rest from further away at a
// half to a sixth of the rate (measured with straight-line code), and the warps of an SM are at different places of their
// solves.  So the loop is written to be short: one copy of the row evaluation serves the start of a descent, the line search
// and the next Newton system (it leaves impulses and curvatures in the head records), one pass over the mass matrix per step
// serves the curvature along the direction and, added up, the inertial force.
//
// The block velocity u and the inertial force M (u - u_free) are carried in double for the descent, updated by the step along
// d and along M d, so that neither has to be recomputed; sums that descend_block compensates in float run in double, one fused
// multiply-add on the FP64 pipe (half the FP32 rate on this GPU) in place of ten FP32 operations.
template <int NR>
NKB_DEV void descend_tree(Env& e, Tile& tile, bool position) {
    const TemplateView& t = *e.t;
    const uint32_t l = e.lane, nb = tile.nblocks, b = t.B, dim = t.ndof;
    const uint32_t* inc = blk_inc(e, nb);
    const uint32_t ib = blk_inc_begin(e, nb, b), ie = blk_inc_begin(e, nb, b + 1u);
    if (position && ib == ie) return;
    const uint32_t chunks = (dim + 3u) >> 2, js = chunks << 2;
    float* velocity = block_vel(e, b, position);
    double* wide = reinterpret_cast<double*>(sm_vec(e, kVecS0));       // spans S0 and S1
    float* flat = sm_vec(e, kVecS2);
    const bool floating = t.floating_root != 0u;
    constexpr int kLevels = kSolveLevels<NR>;
    TreeLane<kLevels> tl;
    if (e.branching) tl = merged_lane<kLevels>(e); else tl = tree_lane<kLevels>(e);
    bool coupled = false;
#pragma unroll 1
    for (uint32_t k = ib + l; k < ie; k += 32u) {
        const uint32_t h = inc[k];
        const uint32_t o = hu(e, HF_OWNER, h);
        coupled |= (o & 0xffffu) != kNoBlock16 && (o >> 16) != kNoBlock16;
        hst3(e, HF_MOVE, h, mk3(0.f, 0.f, 0.f)); hst3(e, HF_STEP, h, mk3(0.f, 0.f, 0.f));
    }
    coupled = __any_sync(NKB_FULL, coupled);
    // the first trip (step -1) only finds M (u - u_free) and the rows where the block stands; Newton steps from 0 on
    int step = -1;
    bool coord[NR];
    double u[NR], dir[NR], inertial[NR];
    float force[NR], fixed[NR];
    const uint32_t half = ie - ib <= 1u ? 0u : min(16u, 1u << (31 - __clz(ie - ib - 1u)));        // of the lanes with a head
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const uint32_t c = l + 32u * r;
        coord[r] = c < dim;
        u[r] = coord[r] ? velocity[c] : 0.0;
        const double fr = coord[r] && !position ? (double)block_free(e, b)[c] : 0.0;
        dir[r] = u[r] - fr;
        inertial[r] = 0.0; force[r] = 0.f;
        fixed[r] = position || !coord[r] ? 0.f : sm_fixed(e)[c];
    }
    bool failure = false;
    float primal = FLT_MAX;
    tick(e, 15);
#pragma unroll 1
    for (;;) {
        // ---- M d, the line's quadratic part ----
        __syncwarp();
#pragma unroll
        for (int r = 0; r < NR; ++r) { wide[l + 32u * r] = dir[r]; flat[l + 32u * r] = (float)dir[r]; }
        __syncwarp();
        double md[NR], sums[4] = {0.0, 0.0, 0.0, 0.0};             // along d: curvature, inertial slope, force, constant impulses
        float fixed_size = 0.f;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            md[r] = coord[r] ? mass_row_times(e, l + 32u * r, chunks, wide) : 0.0;
            sums[0] = fma(dir[r], md[r], sums[0]);
            sums[1] = fma(inertial[r], dir[r], sums[1]);
            sums[2] = fma((double)force[r], dir[r], sums[2]);
            sums[3] = fma((double)fixed[r], dir[r], sums[3]);
            fixed_size = fmaf(fabsf(fixed[r]), fabsf((float)dir[r]), fixed_size);
        }
        bool search = step >= 0;
        double icurv = 0.0, islope = 0.0;
        float initial = 0.f, alpha = 0.f;
        if (search) {
#pragma unroll
            for (int k = 0; k < 4; ++k) sums[k] = warp_sum(sums[k]);
            fixed_size = warp_sum(fixed_size);
            icurv = sums[0];
            // d solves H d = force, so the slope at alpha = 0 is -(force . d)
            initial = -(float)sums[2];
            islope = sums[1];
            if (!isfinite(initial) || !(fabs(islope) <= FLT_MAX) || !(icurv <= FLT_MAX)) { failure = true; break; }
            if (!(initial < 0.f)) break;
            alpha = 1.f;
            tick(e, 20);
            row_steps(e, inc, ib, ie, dim, flat);
            tick(e, 21);
        } else {
#pragma unroll
            for (int r = 0; r < NR; ++r) inertial[r] = md[r];
        }
        // ---- exact line search (block_descent_tile.cuh:2048-2125); without a search one evaluation at the start ----
        {
            float low = 0.f, high = 0.f;
            bool bounded = false;
            int trials = 0;
#pragma unroll 1
            for (;;) {
                double rows; float curvature, magnitude;
                evaluate_line(e, inc, ib, ie, half, alpha, rows, curvature, magnitude);
                tick_count(e, 28);
                if (!search) break;
                const float slope = (float)(islope + (double)alpha * icurv - (rows + sums[3]));
                curvature += (float)icurv;
                magnitude += fabsf((float)islope) + alpha * (float)icurv + fixed_size;
                bool give_up = ++trials >= (int)kLineSteps;
                if (isfinite(slope) && isfinite(curvature)) {
                    if (fabsf(slope) <= fmaxf(kLineTol * -initial, kRoundings * FLT_EPSILON * magnitude)) break;
                    if (slope < 0.f) low = alpha; else { high = alpha; bounded = true; }
                    give_up |= bounded && high - low <= FLT_EPSILON * high;
                    const float next = alpha - __fdividef(slope, curvature);
                    alpha = next > low && (!bounded || next < high) ? next : bounded ? 0.5f * (low + high) : 2.0f * alpha;
                } else { high = alpha; bounded = true; alpha = 0.5f * (low + high); }
                if (give_up) { alpha = low; search = false; }       // one more evaluation, at the point returned
            }
        }
        tick(e, 22);
        tick_count(e, 23);
        // ---- take the step ----
        bool fin = true, rounded = true;
        float longest = 0.f;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const double after = fma((double)alpha, step < 0 ? 0.0 : dir[r], u[r]);
            fin &= fabs(after) <= FLT_MAX;
            rounded &= (float)after == (float)u[r];
            longest = fmaxf(longest, fabsf(alpha * (float)dir[r]));
        }
        if (step >= 0 && !__all_sync(NKB_FULL, fin)) { failure = true; break; }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            u[r] = fma((double)alpha, step < 0 ? 0.0 : dir[r], u[r]);
            inertial[r] = fma((double)alpha, step < 0 ? 0.0 : md[r], inertial[r]);
            force[r] = 0.f;
        }
        if (alpha != 0.f)
#pragma unroll 1
            for (uint32_t k = ib + l; k < ie; k += 32u) {
                const uint32_t h = inc[k];
                const float4 s = hq(e, HF_STEP, h), m = hq(e, HF_MOVE, h);
                hq(e, HF_MOVE, h) = make_float4(fmaf(alpha, s.x, m.x), fmaf(alpha, s.y, m.y), fmaf(alpha, s.z, m.z), m.w);
            }
        if (step >= 0) {
            rounded = __all_sync(NKB_FULL, rounded);
            primal = rounded ? 0.f : warp_max_positive(longest);
            if (!(alpha > 0.f) || rounded || step + 1 == (int)kNewtonSteps) break;
        }
        ++step;
        // ---- the next Newton system at the new velocity: this lane's row of H, its entry of the force balance ----
        __syncwarp();
#pragma unroll
        for (int r = 0; r < NR; ++r) flat[l + 32u * r] = (float)u[r];
        TreeRow<kLevels> row;
        tree_load_row(e, tl, sm_mass(e), e.lay->ld, row);
        float base_row[kTreeBase];
        if (NR > 1) {
#pragma unroll
            for (int k = 0; k < kTreeBase; ++k) base_row[k] = floating && l < 6u ? sm_mass(e)[l * e.lay->ld + k] : 0.f;
        }
        double g[NR];
        float scale[NR], diag[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            g[r] = -inertial[r]; scale[r] = fabsf((float)inertial[r]); diag[r] = 0.f;
            // rows on a single coordinate only touch that coordinate (block_descent_tile.cuh:1555-1568)
            if (tile.units)
#pragma unroll 1
                for (uint32_t slot = 0u; slot < 3u; ++slot) {
                    const uint32_t h = unit_table(e, nb)[slot * e.vstride + l + 32u * r];
                    if (h == kNoUnitHead) continue;
                    const float v = hf(e, HF_UNITV, h);
                    diag[r] += v * hf(e, HF_C, h) * v;
                    g[r] = fma((double)v, (double)hf(e, HF_F, h), g[r]);
                    scale[r] += fabsf(v) * hf(e, HF_NZ, h);
                }
            g[r] += (double)fixed[r]; scale[r] += fabsf(fixed[r]);
        }
        const int depth = (int)tl.depth;
        __syncwarp();
        tick(e, 16);
#pragma unroll 1
        for (uint32_t k = ib; k < ie; ++k) {
            const uint32_t h = inc[k];
            const uint32_t jo = hu(e, HF_JOFF, h);
            if (jo & kUnitRow) break;                        // contact heads come first
            const float4 f = hq(e, HF_F, h), c4 = hq(e, HF_C + 1u, h);
            const float2 nz = *reinterpret_cast<const float2*>(&hf(e, HF_NZ + 1u, h));
            const float c0 = f.w, c1 = c4.x, c2 = c4.y, c12 = c4.z;
            if (c0 + c1 + c2 + c4.w + nz.x + nz.y == 0.f) continue;        // no impulse, no stiffness
            const float* jr = sm_jpool(e) + jo;
            float a0 = 0.f, a1 = 0.f, a2 = 0.f, b0 = 0.f, b1 = 0.f, b2 = 0.f;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const uint32_t c = l + 32u * r;
                const float j0 = coord[r] ? jr[c] : 0.f, j1 = coord[r] ? jr[js + c] : 0.f, j2 = coord[r] ? jr[2u * js + c] : 0.f;
                g[r] = fma((double)j0, (double)f.x, g[r]); g[r] = fma((double)j1, (double)f.y, g[r]); g[r] = fma((double)j2, (double)f.z, g[r]);
                scale[r] += fabsf(j0) * c4.w + fabsf(j1) * nz.x + fabsf(j2) * nz.y;
                const float p0 = j0 * c0, p1 = j1 * c1 + j2 * c12, p2 = j2 * c2 + j1 * c12;
                diag[r] += p0 * j0 + p1 * j1 + p2 * j2;
                if (r == 0) { a0 = b0 = p0; a1 = b1 = p1; a2 = b2 = p2; }
                else if (l < 6u) { a0 = p0; a1 = p1; a2 = p2; }
            }
            if (floating) {
                const float4 x = *reinterpret_cast<const float4*>(jr), y = *reinterpret_cast<const float4*>(jr + js), z = *reinterpret_cast<const float4*>(jr + 2u * js);
                const float2 x2 = *reinterpret_cast<const float2*>(jr + 4), y2 = *reinterpret_cast<const float2*>(jr + js + 4), z2 = *reinterpret_cast<const float2*>(jr + 2u * js + 4);
                row.base[0] += a0 * x.x + a1 * y.x + a2 * z.x; row.base[1] += a0 * x.y + a1 * y.y + a2 * z.y;
                row.base[2] += a0 * x.z + a1 * y.z + a2 * z.z; row.base[3] += a0 * x.w + a1 * y.w + a2 * z.w;
                row.base[4] += a0 * x2.x + a1 * y2.x + a2 * z2.x; row.base[5] += a0 * x2.y + a1 * y2.y + a2 * z2.y;
                if (NR > 1) {
                    base_row[0] += b0 * x.x + b1 * y.x + b2 * z.x; base_row[1] += b0 * x.y + b1 * y.y + b2 * z.y;
                    base_row[2] += b0 * x.z + b1 * y.z + b2 * z.z; base_row[3] += b0 * x.w + b1 * y.w + b2 * z.w;
                    base_row[4] += b0 * x2.x + b1 * y2.x + b2 * z2.x; base_row[5] += b0 * x2.y + b1 * y2.y + b2 * z2.y;
                }
            }
#pragma unroll
            for (int p = 0; p < kLevels; p += 2) {
                if (p >= depth - 1) break;
#pragma unroll
                for (int q = p; q < p + 2; ++q) {
                    const uint32_t at = tl.ancestor(q);
                    row.limb[q] += a0 * jr[at] + a1 * jr[js + at] + a2 * jr[2u * js + at];
                }
            }
        }
        tick(e, 17);
        // the rounding scale: force terms, and what the row's own stiffness makes of the velocities along its root path
        const bool high = NR > 1 && l < 6u && floating;          // this lane's joint is its second coordinate
        row.diag += high ? diag[NR - 1] : diag[0];
        {
            float path = fabsf(row.diag * flat[tl.coord]);
            if (floating) {
                const float4 v = *reinterpret_cast<const float4*>(flat);
                const float2 v2 = *reinterpret_cast<const float2*>(flat + 4);
                path += fabsf(row.base[0] * v.x) + fabsf(row.base[1] * v.y) + fabsf(row.base[2] * v.z) + fabsf(row.base[3] * v.w) + fabsf(row.base[4] * v2.x) + fabsf(row.base[5] * v2.y);
                if (NR > 1)
                    scale[0] += high ? fabsf(base_row[0] * v.x) + fabsf(base_row[1] * v.y) + fabsf(base_row[2] * v.z) + fabsf(base_row[3] * v.w) + fabsf(base_row[4] * v2.x) + fabsf(base_row[5] * v2.y) : 0.f;
            }
            if (high) scale[NR - 1] += path; else scale[0] += path;
        }
        bool finite = true, small = true;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            force[r] = coord[r] ? (float)g[r] : 0.f;
            finite &= isfinite(force[r]);
            small &= !coord[r] || fabsf(force[r]) <= kRoundings * FLT_EPSILON * scale[r];
        }
        if (!__all_sync(NKB_FULL, finite)) { failure = true; break; }
        bool converged = __all_sync(NKB_FULL, small);
        if (converged && tile.tol > 0.f) {
            float d[NR];
            solve_block_mass<NR>(e, b, force, d);
            bool still = true;
#pragma unroll
            for (int r = 0; r < NR; ++r) still &= !coord[r] || fabsf(d[r]) < tile.tol;
            converged = __all_sync(NKB_FULL, still);
        }
        if (converged) { primal = 0.f; break; }
        tick(e, 18);
        // ---- d = H^-1 g ----
        if (NR == 1) {
#pragma unroll
            for (int k = 0; k < kTreeBase; ++k) base_row[k] = row.base[k];
        }
        float x, base_x[kTreeBase];
        if (!tree_solve<NR, false, kLevels>(e, tl, row, high ? force[NR - 1] : force[0], base_row, force[0], e.sm + e.lay->chol, x, base_x)) { failure = true; break; }
        float d[NR];
        tree_scatter<NR>(e, x, base_x, d);
#pragma unroll
        for (int r = 0; r < NR; ++r) dir[r] = d[r];
        tick(e, 19);
    }
    __syncwarp();
#pragma unroll 1
    for (uint32_t k = ib + l; k < ie; k += 32u) {
        const uint32_t h = inc[k];
        const float4 res = hq(e, HF_RES, h), move = hq(e, HF_MOVE, h);
        hq(e, HF_RES, h) = make_float4(__fsub_rn(res.x, move.x), __fsub_rn(res.y, move.y), __fsub_rn(res.z, move.z), res.w);
    }
    if (failure) e.status |= kStatusSolverFailure;
    float moved = failure ? FLT_MAX : 0.f;
#pragma unroll
    for (int r = 0; r < NR; ++r)
        if (coord[r]) {
            const float now = (float)u[r], before = velocity[l + 32u * r];
            moved = fmaxf(moved, residual_abs(now - before));
            velocity[l + 32u * r] = now;
        }
    moved = warp_max_positive(moved);
    tile.momentum = fmaxf(tile.momentum, moved);
    if (failure) primal = FLT_MAX;
    tile.residual = fmaxf(tile.residual, fmaxf(primal, coupled ? moved : 0.f));
    __syncwarp();
}

// The articulation's descent in the space of its rows (nkb_rowspace.cuh): the same model, laws, line search and stopping rules as
// descend_tree, with a lane to a row.  The first descent of a step starts from the multipliers that the heads start from, whatever the
// block's velocity is; the later ones from the multipliers that the last one left.
// A force counts as zero within kRoundings of the rows' terms, and where it moves no coordinate by the velocity tolerance.  Sixteen roundings, about
// what the wider terms of a descent in coordinates allow, left results 6 % further from 64 bits (2048 humanoids, one step; 2 % faster).
template <int NR>
NKB_DEV bool descend_rows(Env& e, Tile& tile, bool position) {
    const TemplateView& t = *e.t;
    const uint32_t l = e.lane, b = t.B, n = t.ndof, m = e.rows;
    const bool fresh = !position && e.by_rows == kRowsFresh;
    float* velocity = block_vel(e, b, position);
    double* wide = reinterpret_cast<double*>(sm_vec(e, kVecS0));       // spans S0 and S1
    RowLane a = {false, false, l, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    bool coupled = false;
    uint32_t h = 0u, axis = 0u;
    if (l < m) {
        const uint32_t entry = row_table(e)[l], owner = hu(e, HF_OWNER, entry & 0xffffu);
        h = entry & 0xffffu; axis = entry >> 16;
        a.live = ((owner & 0xffffu) == b || (owner >> 16) == b) && (axis == 0u || (hu(e, HF_FLAGS, h) & kHeadScalar) == 0u);
        coupled = a.live && (owner & 0xffffu) != kNoBlock16 && (owner >> 16) != kNoBlock16;
        a.tangent = axis != 0u;
        if (a.tangent) a.partner = axis == 1u ? l + 1u : l - 1u;
        const float4 dual = hq(e, HF_DUAL, h), res = hq(e, HF_RES, h);
        a.dual = axis == 0u ? dual.x : axis == 1u ? dual.y : dual.z;
        a.res = axis == 0u ? res.x : axis == 1u ? res.y : res.z;
        a.rho = dual.w; a.lower = hf(e, HF_LOWER, h); a.upper = hf(e, HF_UPPER, h);
        // the friction cone's radius follows the head's normal multiplier at the start of the descent
        a.radius = res.w > 0.f ? (dual.x < 0.0f ? 0.0f : dual.x) * res.w : 0.f;
    }
    const uint32_t live = __ballot_sync(NKB_FULL, a.live);
    coupled = __any_sync(NKB_FULL, coupled);
    if (live == 0u && !fresh) {                     // nothing holds the block: it is where it ends
        return true;
    }
    double y = a.live ? (fresh ? (a.rho > 0.f ? (double)a.dual : 0.0) : row_y(e)[l]) : 0.0;
    float move = 0.f;
    double begin = y;
    double travel[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) travel[r] = 0.0;
    if (fresh) {
        // from the block's velocity to the one that these multipliers give it
        row_spread<NR>(e, m, y, travel);
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const uint32_t c = l + 32u * r;
            if (c < n) travel[r] += (double)row_x(e)[m * t.row_stride + c] - ((double)velocity[c] - (double)block_free(e, b)[c]);
            wide[c] = travel[r];
        }
        __syncwarp();
        if (a.live) move = (float)row_dot(e, h, axis, wide);
    }
    // X and W carry the factor's rounding, and the first descent of a step travels furthest on them: where its rows have settled, what the block's
    // balance lacks in 64 bits moves the block and the rows, which settle again from there.  One step of 2048 humanoids against 64 bits, geometric
    // mean: 6.0e-7, 6.7e-7 without, 6.6e-7 in coordinates; 1970 us for four steps, 1870 without.  In every descent (2620 us) it gives no more.
    bool balanced = !fresh;
    auto balance = [&]() {
        const uint32_t n4 = (n + 3u) & ~3u;
        double lack[NR];
        row_spread<NR>(e, m, a.live ? y - begin : 0.0, travel);
        begin = y;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            const uint32_t c = l + 32u * k;
            wide[c] = c < n ? (double)velocity[c] + travel[k] - (position ? 0.0 : (double)block_free(e, b)[c]) : 0.0;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < NR; ++k) {
            const uint32_t c = l + 32u * k;
            lack[k] = c < n ? (position ? 0.0 : (double)sm_fixed(e)[c]) - mass_row_times(e, c, n4 >> 2, wide) : 0.0;
        }
#pragma unroll 1
        for (uint32_t j = 0u; j < m; ++j) {
            const double yj = __shfl_sync(NKB_FULL, a.live ? y : 0.0, j);
            const uint32_t entry = row_table(e)[j], jo = hu(e, HF_JOFF, entry & 0xffffu);
#pragma unroll
            for (int k = 0; k < NR; ++k) {
                const uint32_t c = l + 32u * k;
                if (c >= n) continue;
                if (!(jo & kUnitRow)) lack[k] = fma((double)sm_jpool(e)[jo + (entry >> 16) * n4 + c], yj, lack[k]);
                else if (c == (jo & 0xffffu)) lack[k] = fma((double)hf(e, HF_UNITV, entry & 0xffffu), yj, lack[k]);
            }
        }
        float force[NR], dir[NR];
#pragma unroll
        for (int k = 0; k < NR; ++k) { force[k] = (float)lack[k]; dir[k] = 0.f; }
        solve_block_mass<NR>(e, b, force, dir);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < NR; ++k) { if (l + 32u * k < n) travel[k] += (double)dir[k]; wide[l + 32u * k] = l + 32u * k < n ? travel[k] : 0.0; }
        __syncwarp();
        if (a.live) move = (float)row_dot(e, h, axis, wide);
        __syncwarp();
    };
    const uint32_t half = m <= 1u ? 0u : min(16u, 1u << (31 - __clz(m - 1u)));         // of the lanes with a row
    bool failure = false, settled = false, stuck = false, last = false;
    float primal = FLT_MAX;
    RowResponse at = row_respond(a, move);
    tick(e, 15);
    float dy = 0.f, alpha = 0.f;
    int step = 0;
#pragma unroll 1
    for (;; ++step) {
        const float r = a.live ? (float)((double)at.impulse - y) : 0.f;
        const float noise = fabsf(at.impulse) + fabsf((float)y) + at.curvature * (fabsf(a.res) + fabsf(move));
        if (!__all_sync(NKB_FULL, isfinite(r) && isfinite(noise))) { failure = true; break; }
        settled = __all_sync(NKB_FULL, fabsf(r) <= kRoundings * FLT_EPSILON * noise);
        if (settled) {
            double d[NR];
            float longest = 0.f;
#pragma unroll
            for (int k = 0; k < NR; ++k) d[k] = 0.0;
            if (tile.tol > 0.f) {
                row_spread<NR>(e, m, (double)r, d);
#pragma unroll
                for (int k = 0; k < NR; ++k) longest = fmaxf(longest, fabsf((float)d[k]));
                longest = warp_max_positive(longest);
            }
            if (!(tile.tol > 0.f) || longest < tile.tol) { primal = 0.f; last = true; }
        }
        if (last) {
            if (balanced) break;
            balance();
            balanced = true; last = step >= (int)kNewtonSteps;
            at = row_respond(a, move);
            --step;
            continue;
        }
        tick(e, 17);
        // ---- (1 + C W) dy = r ----
        const float s = row_product(e, m, r);
        float ra = at.curvature >= FLT_MIN ? at.curvature * rsqrt_normal(at.curvature) : 0.f, rb = 0.f;
        if (__any_sync(NKB_FULL, at.cross != 0.f)) {
            const float other = __shfl_sync(NKB_FULL, ra, a.partner);
            if (at.cross != 0.f) { if (axis == 1u) rb = copysignf(other, at.cross); else ra = 0.f; }
        }
        if (!solve_rows<kRowGroups>(e, m, a.partner, ra, rb, r, s, dy)) { failure = true; break; }
        tick(e, 19);
        const float along = row_product(e, m, dy);
        double decrement = (double)r * (double)along;
        float icurv = dy * along, unused = 0.f;
        line_sums(decrement, icurv, unused, half, l);
        const float initial = -(float)decrement;
        if (!isfinite(initial) || !(icurv <= FLT_MAX)) { failure = true; break; }
        tick(e, 20);
        // ---- exact line search (block_descent_tile.cuh:2048-2125) ----
        const float aside = __shfl_sync(NKB_FULL, along, a.partner);
        // rows that hold one another (W r = 0) share their load anew without moving the block: a whole step, nothing to search
        bool search = initial < 0.f, bounded = false;
        float low = 0.f, high = 0.f;
        int trials = 0;
        alpha = 1.f;
#pragma unroll 1
        for (;;) {
            const float trial = fmaf(alpha, along, move);
            const double ahead = fma((double)alpha, (double)dy, y);
            at = row_respond(a, trial);
            tick_count(e, 28);
            double slope64 = (ahead - (double)at.impulse) * (double)along;
            float curvature = fmaf(at.curvature, along, at.cross * aside) * along;
            float magnitude = (fabsf(at.impulse) + fabsf((float)ahead) + kImpulseRounding * at.curvature * (fabsf(a.res) + fabsf(trial))) * fabsf(along);
            if (!a.live) { slope64 = 0.0; curvature = 0.f; magnitude = 0.f; }
            line_sums(slope64, curvature, magnitude, half, l);
            if (!search) break;
            const float slope = (float)slope64;
            curvature += icurv;
            bool give_up = ++trials >= (int)kLineSteps;
            if (isfinite(slope) && isfinite(curvature)) {
                if (fabsf(slope) <= fmaxf(kLineTol * -initial, kRoundings * FLT_EPSILON * magnitude)) break;
                if (slope < 0.f) low = alpha; else { high = alpha; bounded = true; }
                give_up |= bounded && high - low <= FLT_EPSILON * high;
                const float next = alpha - __fdividef(slope, curvature);
                alpha = next > low && (!bounded || next < high) ? next : bounded ? 0.5f * (low + high) : 2.0f * alpha;
            } else { high = alpha; bounded = true; alpha = 0.5f * (low + high); }
            if (give_up) { alpha = low; search = false; }       // one more evaluation, at the point returned
        }
        tick(e, 22);
        tick_count(e, 23);
        // ---- take the step ----
        const double after = fma((double)alpha, (double)dy, y);
        const bool rounded = __all_sync(NKB_FULL, after == y);
        y = after; move = fmaf(alpha, along, move);
        if (!(alpha > 0.f) || rounded || settled || step + 1 == (int)kNewtonSteps) {
            double d[NR];
            float longest = 0.f;
#pragma unroll
            for (int k = 0; k < NR; ++k) d[k] = 0.0;
            row_spread<NR>(e, m, (double)(alpha * dy), d);
#pragma unroll
            for (int k = 0; k < NR; ++k) longest = fmaxf(longest, fabsf((float)d[k]));
            primal = rounded ? 0.f : warp_max_positive(longest);
            stuck = !settled && step + 1 == (int)kNewtonSteps;
            last = !settled || !(alpha > 0.f) || rounded || primal < tile.tol || step + 1 == (int)kNewtonSteps;
        }
    }
    // ---- the block's velocity and its rows' residuals at the multipliers found ----
    if (failure) e.status |= kStatusSolverFailure;
    row_spread<NR>(e, m, a.live ? y - begin : 0.0, travel);
    float moved = failure ? FLT_MAX : 0.f;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const uint32_t c = l + 32u * r;
        wide[c] = c < n ? travel[r] : 0.0;
        if (c < n) {
            const float before = velocity[c], now = (float)((double)before + travel[r]);
            moved = fmaxf(moved, residual_abs(now - before));
            velocity[c] = now;
        }
    }
    __syncwarp();
    if (a.live) {
        hf(e, HF_RES + axis, h) = (float)((double)a.res - row_dot(e, h, axis, wide));
        row_y(e)[l] = y;
    }
    if (!position) e.by_rows = kRowsSettled;
    moved = warp_max_positive(moved);
    tile.momentum = fmaxf(tile.momentum, moved);
    if (failure) primal = FLT_MAX;
    if (!stuck) tile.residual = fmaxf(tile.residual, fmaxf(primal, coupled ? moved : 0.f));
    __syncwarp();
    return !stuck;
}

// ---- team mode: several warps on one env ---------------------------------------------------------------------------------
// Blocks of one colour share no constraint row (index_blocks colours the graph whose edges are the two-sided heads), so
// their descents touch disjoint head records and disjoint body velocities and may run side by side.  The env's lead warp
// walks the descent order; for a run of rigid blocks of one colour it publishes a command in shared memory, and every
// warp of the team (the lead included) takes its share of the run, four blocks at a time, in registers
// (descend_bodies).  A result does not depend on which warp ran a block, so team sizes give bit-identical states.
//
// The warps meet through sequence numbers in shared memory, never through a hardware barrier: the lead bumps the
// command's sequence number, a helper answers by copying it into its result record.  Every wait is bounded by a cycle
// budget; a warp whose wait runs out records kStatusTeamTimeout and carries on alone (the lead descends the remaining
// blocks itself, a helper leaves), so a team that falls apart costs a status bit, not a hung kernel.
enum : uint32_t { kTeamDescend = 0x44455343u, kTeamExit = 0x45584954u,
                  // stages whose outer loop is dealt out over the team: k_begin carries the stage's count argument
                  kTeamNarrowphase = 0x4e415252u, kTeamWarmStart = 0x5741524du, kTeamCacheOwners = 0x4f574e52u };
constexpr uint32_t kTeamCommandWords = 12u;                   // the team area: command, then 4 result words per member
constexpr long long kTeamPatience = 4000000000ll;           // cycles a warp waits for another: about two seconds
struct TeamCommand { uint32_t seq, op, k_begin, k_end, position, nblocks, nheads; float tol; uint32_t dead, pad0, pad1, pad2; };
static_assert(sizeof(TeamCommand) == 4u * kTeamCommandWords, "the command occupies the first words of the team area");

NKB_DEV TeamCommand* team_command(float* sm, const SmemLayout& lay) { return reinterpret_cast<TeamCommand*>(sm + lay.team_area); }
// result record of a member: momentum, residual, status, sequence number of the last command it finished
NKB_DEV float* team_result(float* sm, const SmemLayout& lay, uint32_t member) { return sm + lay.team_area + kTeamCommandWords + 4u * member; }
NKB_DEV uint32_t team_peek(const uint32_t* word) { return *reinterpret_cast<const volatile uint32_t*>(word); }
NKB_DEV void team_poke(uint32_t* word, uint32_t value) { *reinterpret_cast<volatile uint32_t*>(word) = value; }

// Lead warp, before any helper looks: sequence numbers start at zero (called by every team's lead ahead of a block-wide
// barrier at kernel start).
NKB_DEV void team_open(float* sm, const SmemLayout& lay, uint32_t lane) {
    TeamCommand* cmd = team_command(sm, lay);
    if (lane == 0u) { cmd->seq = 0u; cmd->op = 0u; cmd->dead = 0u; }
    if (lane < lay.team) reinterpret_cast<uint32_t*>(team_result(sm, lay, lane))[3] = 0u;
}

// Lead warp: publishes a command; returns its sequence number.
NKB_DEV uint32_t team_post(float* sm, const SmemLayout& lay, uint32_t lane, uint32_t op, uint32_t k_begin, uint32_t k_end, bool position, const Tile& tile) {
    TeamCommand* cmd = team_command(sm, lay);
    __syncwarp();
    const uint32_t seq = cmd->seq + 1u;
    __syncwarp();
    if (lane == 0u) {
        cmd->op = op; cmd->k_begin = k_begin; cmd->k_end = k_end; cmd->position = position ? 1u : 0u;
        cmd->nblocks = tile.nblocks; cmd->nheads = tile.nheads; cmd->tol = tile.tol;
        __threadfence_block();
        team_poke(&cmd->seq, seq);
    }
    __syncwarp();
    return seq;
}

// Lead warp: waits until every helper has answered command `seq`; false when the budget ran out.
NKB_DEV bool team_collect(float* sm, const SmemLayout& lay, uint32_t lane, uint32_t seq) {
    // every lane polls the same word, so the warp never splits over a wait
    bool answered = true;
    const long long begin = clock64();
#pragma unroll 1
    for (uint32_t m = 1u; m < lay.team && answered; ++m) {
        const uint32_t* done = reinterpret_cast<const uint32_t*>(team_result(sm, lay, m)) + 3;
#pragma unroll 1
        while (team_peek(done) != seq) {
            if (clock64() - begin > kTeamPatience) { answered = false; break; }
            __nanosleep(40);
        }
    }
    answered = __all_sync(NKB_FULL, answered);
    __threadfence_block();
    return answered;
}

// An env record for a warp that works on an env's shared-memory slice without owning its articulation lanes (a team's
// helper): pointers and lane only, no link or coordinate state.
NKB_DEV Env bare_env(float* sm, const SmemLayout* lay, const TemplateView* t, const StateView* s, uint32_t env, uint32_t lane, uint32_t vstride) {
    Env e;
    e.t = t; e.s = s; e.lay = lay; e.sm = sm; e.env = env; e.lane = lane;
    e.parent = kNoLink; e.jtype = kFixed; e.depth = 0xffffu; e.link_dof = 0u;
    e.q = e.qd = e.qdd = e.tau = 0.f;
    e.axis = mk3(0.f, 0.f, 0.f);
    e.drive_command = e.drive_dissipation = e.drive_lower = e.drive_upper = 0.f;
    e.dof_link[0] = e.dof_link[1] = 0u; e.dof_comp[0] = e.dof_comp[1] = kNoLink;
    e.status = 0u; e.branching = false; e.merged = kMergeUntried; e.by_rows = kRowsNone; e.rows = 0u; e.reach = 0u; e.pool = sm + lay->jpool; e.vstride = vstride;
#ifdef NKB_STAGE_TAPS
    e.cyc = nullptr; e.t0 = 0;
#endif
    return e;
}

// What a warp needs to descend rigid blocks.
struct RigidRun {
    float* sm;
    const SmemLayout* lay;
    const TemplateView* t;
    uint32_t lane, vstride;
    uint32_t nheads, nblocks;
    float tol;
};
struct RigidResult { float momentum, residual; uint32_t status; };

// A warp works on four free bodies at once, eight lanes on each: blocks of one colour share no constraint row.  Inside a group a
// lane is a constraint row in the line search (rows j, j + 8, ...) and a row of the 6 x 6 Newton system in its assembly; everything
// of the block's own size (its velocity, its mass, the factorisation) is replicated over the group's lanes in registers, so that
// neither shared memory nor an exchange sits inside those chains.  Loops run until the last group of the warp is done; a group that
// is done leaves its state alone.  A body of a 48-box pile has 3.5 rows: sixteen lanes to a body, two bodies to a warp, kept twice the
// warps busy with the same instructions (1024 such piles 20.1 ms, eight lanes 15.5; 700 of 24 boxes 8.07 and 5.85).
constexpr uint32_t kBodyLanes = 8u, kBodyGroups = 32u / kBodyLanes;
struct BodyLanes {
    uint32_t j, mask, first;             // lane within the group, the group's lanes, its first lane
    NKB_DEV bool any(bool p) const { return (__ballot_sync(NKB_FULL, p) & mask) != 0u; }
    NKB_DEV bool all(bool p) const { return (__ballot_sync(NKB_FULL, p) & mask) == mask; }
    // v[k] summed over the group's lanes, dealt out: lane j gets the sums of v[j N / 8 ...] in v[0 .. N / 8).  Each
    // exchange halves what a lane still holds (28 shuffles for 32 values over 8 lanes; a sum per value would take 96)
    template <typename T, int N> NKB_DEV void deal(T (&v)[N]) const {
        int held = N / 2;
#pragma unroll
        for (int o = 4; o > 0; o >>= 1, held >>= 1) {
            const bool upper = (j & o) != 0u;
#pragma unroll
            for (int k = 0; k < held; ++k) {
                const T give = upper ? v[k] : v[k + held], keep = upper ? v[k + held] : v[k];
                v[k] = keep + __shfl_xor_sync(NKB_FULL, give, o);
            }
        }
    }
    template <typename T> NKB_DEV T sum(T v) const {
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(NKB_FULL, v, o);
        return v;
    }
};
NKB_DEV BodyLanes body_lanes(uint32_t lane) {
    BodyLanes g;
    g.j = lane & (kBodyLanes - 1u); g.first = lane & ~(kBodyLanes - 1u);
    g.mask = ((1u << kBodyLanes) - 1u) << g.first;
    return g;
}
// M v of a free body: mass, and the world inertia xx yy zz xy xz yz
struct BodyMass { float m, i[6]; };
NKB_DEV void body_mass_mul(const BodyMass& b, const double (&v)[6], double (&out)[6]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k] = (double)b.m * v[k];
    out[3] = fma((double)b.i[0], v[3], fma((double)b.i[3], v[4], (double)b.i[4] * v[5]));
    out[4] = fma((double)b.i[3], v[3], fma((double)b.i[1], v[4], (double)b.i[5] * v[5]));
    out[5] = fma((double)b.i[4], v[3], fma((double)b.i[5], v[4], (double)b.i[2] * v[5]));
}
// Row j < 6 of a contact's Jacobian is J_ax[j] = dir_ax . w_j with w_j the unit vector for the linear rows and unit x arm for
// the angular ones (dir . (unit x arm) = (arm x dir) . unit); rows 6 and 7 of a group of eight get zeros.
NKB_DEV V3 body_row_axis(uint32_t row, V3 arm) {
    return row == 0u ? mk3(1.f, 0.f, 0.f) : row == 1u ? mk3(0.f, 1.f, 0.f) : row == 2u ? mk3(0.f, 0.f, 1.f)
         : row == 3u ? mk3(0.f, -arm.z, arm.y) : row == 4u ? mk3(arm.z, 0.f, -arm.x) : row == 5u ? mk3(-arm.y, arm.x, 0.f) : mk3(0.f, 0.f, 0.f);
}
template <typename T> NKB_DEV T pick6(const T (&v)[6], uint32_t k) { return k == 0u ? v[0] : k == 1u ? v[1] : k == 2u ? v[2] : k == 3u ? v[3] : k == 4u ? v[4] : v[5]; }

// products with their fused multiply-adds spelled out
NKB_DEV float dot_fma(V3 a, V3 b) { return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)); }
NKB_DEV V3 cross_fma(V3 a, V3 b) { return mk3(fmaf(a.y, b.z, -(a.z * b.y)), fmaf(a.z, b.x, -(a.x * b.z)), fmaf(a.x, b.y, -(a.y * b.x))); }

NKB_DEV V3 mix_fma(V3 a, float p, V3 b, float q) { return mk3(fmaf(a.x, p, b.x * q), fmaf(a.y, p, b.y * q), fmaf(a.z, p, b.z * q)); }
// One constraint row J = (n, m), m = arm x n, in a lane's share of a body's Newton system: its impulse's part of the force
// balance and its part of the rounding scale (entry i of which sits in share[4 i + 3], entry k of the lower triangle in
// share[4 (k / 3) + k % 3]: dealt out over eight lanes, lane i gets row i's scale and three entries of the matrix).
NKB_DEV void body_row_share(V3 n, V3 m, float impulse, float size, float (&share)[32], double (&balance)[8]) {
    const float j[6] = {n.x, n.y, n.z, m.x, m.y, m.z};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
        balance[i] = fma((double)j[i], (double)impulse, balance[i]);
        share[4 * i + 3] = fmaf(fabsf(j[i]), size, share[4 * i + 3]);
    }
}
// J (K J)^T of one row: J = (n, m), its row of K J = (p, q)
NKB_DEV void body_block_share(V3 n, V3 m, V3 p, V3 q, float (&share)[32]) {
    const float j[6] = {n.x, n.y, n.z, m.x, m.y, m.z}, c[6] = {p.x, p.y, p.z, q.x, q.y, q.z};
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int k = 0; k <= i; ++k) {
            const int at = i * (i + 1) / 2 + k;
            share[4 * (at / 3) + at % 3] = fmaf(j[i], c[k], share[4 * (at / 3) + at % 3]);
        }
}

// Descends the rigid blocks order[k_begin ..  k_end) of one colour whose turn falls to this warp: four blocks at a
// time, warp `first` of `stride`.  Same model, stopping rules and exact line search as descend_block; the sums that one
// compensates in float run in double, the inertial force is carried as in descend_tree.
// The 6 x 6 systems are assembled by summing heads per lane and dealing the sums out, in every launch form: a sum's order decides
// its last bits, and an env's state must not depend on the batch that it is in.  A row per lane that walks all heads of its body is
// less code and a longer chain (48-box piles, 1024 envs: 28.7 ms, dealt out 26.9; policy steps of 150 quadrupeds with 6 boxes: 5.29
// and 3.92; 2400 of them, in split steps: 7.72 and 6.70; 4096 with 4 boxes: 7.65 and 7.73).
// What bounds it is the length of the chain of one block (assembly, factorisation, line search).  One block per warp with six
// busy lanes and its matrix in shared memory took about 16 k cycles per block; see the team and box figures at World::BuildLayout.
// Inlined for the lead and for its helpers (out of line it spilled the callers' registers and ran 5 % slower), so every fused
// multiply-add is written as one: left to the compiler, the two copies contracted some products differently, and a block's
// result depended on who ran it.
NKB_DEV RigidResult descend_bodies(const RigidRun& run, uint32_t k_begin, uint32_t k_end, uint32_t first, uint32_t stride, bool position) {
    Env e = bare_env(run.sm, run.lay, run.t, nullptr, 0u, run.lane, run.vstride);
    const TemplateView& t = *e.t;
    const BodyLanes g = body_lanes(e.lane);
    const uint32_t nb = run.nblocks, row = g.j;
    const uint32_t* order = block_order(e, nb);
    float most_moved = 0.f, worst = 0.f;
    bool failed = false;
#pragma unroll 1
    for (uint32_t base = k_begin + first * kBodyGroups; base < k_end; base += stride * kBodyGroups) {
        const uint32_t turn = base + e.lane / kBodyLanes;
        const bool have = turn < k_end;
        const uint32_t b = order[have ? turn : base];
        const uint32_t* inc = blk_inc(e, nb) + blk_inc_begin(e, nb, b);
        const uint32_t count = have ? blk_inc_begin(e, nb, b + 1u) - blk_inc_begin(e, nb, b) : 0u;
        // a block without a push-out row keeps its zero position correction; in the velocity phase an unconstrained block
        // still has to reach its free velocity
        const bool began = have && !(position && count == 0u);
        bool active = began, coupled = false, failure = false;
#pragma unroll 1
        for (uint32_t k = g.j; k < count; k += kBodyLanes) {
            const uint32_t h = inc[k], o = hu(e, HF_OWNER, h);
            coupled |= (o & 0xffffu) != kNoBlock16 && (o >> 16) != kNoBlock16;
            hst3(e, HF_MOVE, h, mk3(0.f, 0.f, 0.f)); hst3(e, HF_STEP, h, mk3(0.f, 0.f, 0.f));
        }
        coupled = g.any(coupled);
        BodyMass mass;
        {
            const float* bm = sm_bmass(e, b);
            mass.m = bm[0];
#pragma unroll
            for (int k = 0; k < 6; ++k) mass.i[k] = bm[1 + k];
        }
        float* velocity = block_vel(e, b, position);
        // the first trip (step -1) only finds M (u - u_free) and the rows where the block stands; Newton steps from 0 on.  Every group
        // is at the same step.
        int step = -1;
        double u[6], dir[6], inertial[6];
        float force[6], primal = FLT_MAX;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const double fr = position ? 0.0 : (double)sm_bfree(e, b)[k];
            u[k] = velocity[k];
            dir[k] = u[k] - fr;
            inertial[k] = 0.0; force[k] = 0.f;
        }
#pragma unroll 1
        for (;;) {
            double md[6];
            body_mass_mul(mass, dir, md);
            bool search = active && step >= 0;
            double icurv = 0.0, islope = 0.0;
            float initial = 0.f, alpha = 0.f;
#pragma unroll
            for (int k = 0; k < 6; ++k) icurv = fma(dir[k], md[k], icurv);
            if (step < 0) {
#pragma unroll
                for (int k = 0; k < 6; ++k) inertial[k] = md[k];
            } else {
                double along = 0.0;
#pragma unroll
                for (int k = 0; k < 6; ++k) { islope = fma(inertial[k], dir[k], islope); along = fma((double)force[k], dir[k], along); }
                initial = -(float)along;                     // d solves H d = force
                const bool sane = isfinite(initial) && fabs(islope) <= FLT_MAX && icurv <= FLT_MAX;
                failure |= active && !sane;
                active = active && sane && initial < 0.f;
                search = active; alpha = 1.f;
            }
            // rows' steps along d: dir . (d_lin + d_ang x arm), signed by the side the block is on
            if (search)
#pragma unroll 1
                for (uint32_t k = g.j; k < count; k += kBodyLanes) {
                    const uint32_t h = inc[k];
                    const bool first_side = (hu(e, HF_OWNER, h) & 0xffffu) == b;
                    const V3 arm = hf3(e, first_side ? HF_RA : HF_RB, h);
                    const V3 ang = mk3((float)dir[3], (float)dir[4], (float)dir[5]);
                    V3 v = mk3((float)dir[0], (float)dir[1], (float)dir[2]) + cross_fma(ang, arm);
                    if (!first_side) v = -v;
                    V3 s = mk3(dot_fma(hf3(e, HF_N, h), v), 0.f, 0.f);
                    if (!position) { s.y = dot_fma(hf3(e, HF_T1, h), v); s.z = dot_fma(hf3(e, HF_T2, h), v); }
                    hst3(e, HF_STEP, h, s);
                }
            // exact line search (block_descent_tile.cuh:2048-2125); groups without a search take one evaluation at the start
            {
                float low = 0.f, high = 0.f;
                bool bounded = false, trying = active;
                int trials = 0;
#pragma unroll 1
                while (__any_sync(NKB_FULL, trying)) {
                    double rows = 0.0;
                    float curvature = 0.f, magnitude = 0.f;
                    if (trying)
#pragma unroll 1
                        for (uint32_t k = g.j; k < count; k += kBodyLanes) evaluate_head(e, inc[k], alpha, rows, curvature, magnitude);
                    __syncwarp();
                    rows = g.sum(rows); curvature = g.sum(curvature); magnitude = g.sum(magnitude);
                    if (!trying) continue;
                    if (!search) { trying = false; continue; }
                    const float slope = (float)(fma((double)alpha, icurv, islope) - rows);
                    curvature += (float)icurv;
                    magnitude += fmaf(alpha, (float)icurv, fabsf((float)islope));
                    bool give_up = ++trials >= (int)kLineSteps;
                    if (isfinite(slope) && isfinite(curvature)) {
                        if (fabsf(slope) <= fmaxf(kLineTol * -initial, kRoundings * FLT_EPSILON * magnitude)) { trying = false; continue; }
                        if (slope < 0.f) low = alpha; else { high = alpha; bounded = true; }
                        give_up |= bounded && high - low <= FLT_EPSILON * high;
                        const float next = alpha - __fdividef(slope, curvature);
                        alpha = next > low && (!bounded || next < high) ? next : bounded ? 0.5f * (low + high) : 2.0f * alpha;
                    } else { high = alpha; bounded = true; alpha = 0.5f * (low + high); }
                    if (give_up) { alpha = low; search = false; }       // one more evaluation, at the point returned
                }
            }
            // take the step
            {
                bool finite = true, rounded = true;
                float longest = 0.f;
                double after[6];
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    after[k] = fma((double)alpha, dir[k], u[k]);
                    finite &= fabs(after[k]) <= FLT_MAX;
                    rounded &= (float)after[k] == (float)u[k];
                    longest = fmaxf(longest, fabsf(alpha * (float)dir[k]));
                }
                if (step >= 0) { failure |= active && !finite; active = active && finite; }
                if (active) {
                    if (alpha != 0.f) {
#pragma unroll
                        for (int k = 0; k < 6; ++k) { u[k] = after[k]; inertial[k] = fma((double)alpha, md[k], inertial[k]); }
#pragma unroll 1
                        for (uint32_t k = g.j; k < count; k += kBodyLanes) {
                            const uint32_t h = inc[k];
                            const float4 s = hq(e, HF_STEP, h), m = hq(e, HF_MOVE, h);
                            hq(e, HF_MOVE, h) = make_float4(fmaf(alpha, s.x, m.x), fmaf(alpha, s.y, m.y), fmaf(alpha, s.z, m.z), m.w);
                        }
                    }
                    if (step >= 0) {
                        primal = rounded ? 0.f : longest;
                        active = alpha > 0.f && !rounded && step + 1 < (int)kNewtonSteps;
                    }
                }
            }
            if (!__any_sync(NKB_FULL, active)) break;
            ++step;
            __syncwarp();
            // the next Newton system: the lower triangle of H, this lane's entry of the force balance and its rounding scale
            float a[21], rhs[6], own, scale;
            // a lane takes the heads j, j + 8, ... and sums its share of everything; the lanes then add their shares
            float share[32];
            double balance[8];
#pragma unroll
            for (int k = 0; k < 32; ++k) share[k] = 0.f;
#pragma unroll
            for (int k = 0; k < 8; ++k) balance[k] = 0.0;
            if (active)
#pragma unroll 1
                for (uint32_t k = g.j; k < count; k += kBodyLanes) {
                    const uint32_t h = inc[k];
                    const bool first_side = (hu(e, HF_OWNER, h) & 0xffffu) == b;
                    const V3 arm = hf3(e, first_side ? HF_RA : HF_RB, h), n = hf3(e, HF_N, h), m0 = cross_fma(arm, n);
                    const float4 f = hq(e, HF_F, h);
                    body_row_share(n, m0, first_side ? f.x : -f.x, hf(e, HF_NZ, h), share, balance);
                    body_block_share(n, m0, n * f.w, m0 * f.w, share);
                    if (!position) {                               // push-out rows have a normal axis only
                        const float4 c = hq(e, HF_C + 1u, h);
                        const float2 nz = *reinterpret_cast<const float2*>(&hf(e, HF_NZ + 1u, h));
                        const V3 t1 = hf3(e, HF_T1, h), t2 = hf3(e, HF_T2, h), m1 = cross_fma(arm, t1), m2 = cross_fma(arm, t2);
                        body_row_share(t1, m1, first_side ? f.y : -f.y, nz.x, share, balance);
                        body_row_share(t2, m2, first_side ? f.z : -f.z, nz.y, share, balance);
                        body_block_share(t1, m1, mix_fma(t1, c.x, t2, c.z), mix_fma(m1, c.x, m2, c.z), share);
                        body_block_share(t2, m2, mix_fma(t2, c.y, t1, c.z), mix_fma(m2, c.y, m1, c.z), share);
                    }
                }
            __syncwarp();
            g.deal(share); g.deal(balance);
            scale = share[3];
            const double inner = pick6(inertial, row);
            own = (float)(balance[0] - (row < 6u ? inner : 0.0));
            scale += row < 6u ? fabsf((float)inner) : 0.f;
#pragma unroll
            for (int k = 0; k < 21; ++k) a[k] = __shfl_sync(NKB_FULL, share[k % 3], g.first + k / 3);
            a[0] = __fadd_rn(a[0], mass.m); a[2] = __fadd_rn(a[2], mass.m); a[5] = __fadd_rn(a[5], mass.m);
            a[9] = __fadd_rn(a[9], mass.i[0]); a[13] = __fadd_rn(a[13], mass.i[3]); a[14] = __fadd_rn(a[14], mass.i[1]);
            a[18] = __fadd_rn(a[18], mass.i[4]); a[19] = __fadd_rn(a[19], mass.i[5]); a[20] = __fadd_rn(a[20], mass.i[2]);
            float reach[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                reach[i] = 0.f;
#pragma unroll
                for (int k = 0; k < 6; ++k) reach[i] = fmaf(fabsf(i >= k ? a[i * (i + 1) / 2 + k] : a[k * (k + 1) / 2 + i]), fabsf((float)u[k]), reach[i]);
            }
            scale += pick6(reach, row);
            const bool finite = g.all(isfinite(own)), small = g.all(row >= 6u || fabsf(own) <= kRoundings * FLT_EPSILON * scale);
            failure |= active && !finite;
            active = active && finite;
            float inv[6], x[6];
#pragma unroll
            for (int i = 0; i < 6; ++i) rhs[i] = force[i] = __shfl_sync(NKB_FULL, own, g.first + i);
            if (active && small) {
                bool still = true;
                if (run.tol > 0.f) {
                    const float im = __ldg(t.inv_mass + b);
                    const float* w = sm_bwinv(e, b);
                    const V3 ang = mk3(dot_fma(mk3(w[0], w[3], w[4]), mk3(force[3], force[4], force[5])), dot_fma(mk3(w[3], w[1], w[5]), mk3(force[3], force[4], force[5])),
                                       dot_fma(mk3(w[4], w[5], w[2]), mk3(force[3], force[4], force[5])));
                    still = fabsf(force[0] * im) < run.tol && fabsf(force[1] * im) < run.tol && fabsf(force[2] * im) < run.tol &&
                            fabsf(ang.x) < run.tol && fabsf(ang.y) < run.tol && fabsf(ang.z) < run.tol;
                }
                if (still) { primal = 0.f; active = false; }
            }
            if (!__any_sync(NKB_FULL, active)) break;
            const bool definite = solve6<false>(a, rhs, inv, x);
            failure |= active && !definite;
            active = active && definite;
#pragma unroll
            for (int k = 0; k < 6; ++k) dir[k] = x[k];
        }
        // the block's rows and velocity go back
        if (began) {
#pragma unroll 1
            for (uint32_t k = g.j; k < count; k += kBodyLanes) {
                const uint32_t h = inc[k];
                const float4 res = hq(e, HF_RES, h), move = hq(e, HF_MOVE, h);
                hq(e, HF_RES, h) = make_float4(__fsub_rn(res.x, move.x), __fsub_rn(res.y, move.y), __fsub_rn(res.z, move.z), res.w);
            }
            float moved = failure ? FLT_MAX : 0.f;
#pragma unroll
            for (int k = 0; k < 6; ++k) moved = fmaxf(moved, residual_abs((float)u[k] - velocity[k]));
            failed |= failure;
            most_moved = fmaxf(most_moved, moved);
            worst = fmaxf(worst, fmaxf(failure ? FLT_MAX : primal, coupled ? moved : 0.f));
        }
        __syncwarp();
        if (began && g.j < 6u) velocity[g.j] = (float)pick6(u, g.j);
        __syncwarp();
    }
    RigidResult out;
    out.momentum = warp_max_positive(most_moved); out.residual = warp_max_positive(worst);
    out.status = __any_sync(NKB_FULL, failed) ? (uint32_t)kStatusSolverFailure : 0u;
    return out;
}

// One copy for the lead and its helpers, where nothing of an articulation sits in the caller's registers (worlds of bodies only):
// their warps fetch the same instructions then (48-box piles: 22.2 ms against 20.4, see World::BuildLayout).
static __device__ __noinline__ RigidResult descend_bodies_call(float* sm, const SmemLayout* lay, const TemplateView* t, uint32_t lane, uint32_t vstride, uint32_t nheads, uint32_t nblocks,
                                                               float tol, uint32_t k_begin, uint32_t k_end, uint32_t first, uint32_t stride, bool position) {
    const RigidRun run = {sm, lay, t, lane, vstride, nheads, nblocks, tol};        // a struct argument would go through memory
    return descend_bodies(run, k_begin, k_end, first, stride, position);
}
template <int NR>
NKB_DEV RigidResult descend_share(const RigidRun& run, uint32_t k_begin, uint32_t k_end, uint32_t first, uint32_t stride, bool position) {
    if constexpr (NR == 0) return descend_bodies_call(run.sm, run.lay, run.t, run.lane, run.vstride, run.nheads, run.nblocks, run.tol, k_begin, k_end, first, stride, position);
    else return descend_bodies(run, k_begin, k_end, first, stride, position);
}

// Lead warp: releases the helpers for good (they need not answer).
NKB_DEV void team_dismiss(float* sm, const SmemLayout& lay, uint32_t lane) {
    if (lay.team <= 1u) return;
    Tile none;
    none.nheads = 0u; none.nblocks = 0u; none.units = false; none.momentum = 0.f; none.residual = 0.f; none.tol = 0.f;
    team_post(sm, lay, lane, kTeamExit, 0u, 0u, false, none);
}

// Lead warp: deals a stage's outer loop out over the team.  `work(first, stride)` is the loop body's range form; the lead
// runs its own share between publishing the command and collecting the answers.  Alone (no team, or a team that fell
// apart) the lead runs the whole range.  Returns the helpers' status bits.
template <typename Work>
NKB_DEV void team_fork(Env& e, uint32_t op, uint32_t count, Work&& work) {
    const uint32_t team = e.lay->team;
    if (team <= 1u || team_command(e.sm, *e.lay)->dead != 0u) { work(0u, 1u); return; }
    Tile none;
    none.nheads = 0u; none.nblocks = 0u; none.units = false; none.momentum = 0.f; none.residual = 0.f; none.tol = 0.f;
    const uint32_t seq = team_post(e.sm, *e.lay, e.lane, op, count, 0u, false, none);
    work(0u, team);
    if (team_collect(e.sm, *e.lay, e.lane, seq)) {
#pragma unroll 1
        for (uint32_t m = 1u; m < team; ++m) e.status |= reinterpret_cast<const uint32_t*>(team_result(e.sm, *e.lay, m))[2];
    } else {
        // a helper did not answer: flag the env, stop using the team, and do the whole range here (the stages dealt out
        // this way write each item from its inputs alone, so items done twice come out the same)
        e.status |= kStatusTeamTimeout;
        if (e.lane == 0u) team_command(e.sm, *e.lay)->dead = 1u;
        __syncwarp();
        work(0u, 1u);
    }
}

// The articulation's block: in the space of its rows; else on its tree, with the branches joined that a contact acts on; dense where that is
// too deep.
template <int NR, bool kRows>
NKB_DEV void descend_articulation(Env& e, Tile& tile, bool position) {
    if constexpr (kRows) {
        if (e.by_rows != 0u) {
            if (descend_rows<NR>(e, tile, position)) return;
            e.by_rows = kRowsNone;                   // from where the rows left the block
        }
    }
    if (e.branching && e.t->merges != 0u && e.merged == kMergeUntried) e.merged = merge_trees<NR>(e, tile.nheads);
    if (e.t->tree_depth != 0u && (!e.branching || (e.t->merges != 0u && e.merged != 0u))) descend_tree<NR>(e, tile, position);
    else descend_block<NR>(e, tile, e.t->B, position);
}

// Blocks descend colour by colour, blocks of one colour in index order (block_descent_tile.cuh:2749-2820).
template <int NR, bool kRigid, bool kRows>
NKB_DEV void descend_blocks(Env& e, Tile& tile, bool position) {
    const uint32_t nb = tile.nblocks;
    const uint32_t* order = block_order(e, nb);
    const uint32_t count = order[nb];
    if constexpr (!kRigid) {
#pragma unroll 1
        for (uint32_t k = 0u; k < count; ++k) descend_articulation<NR, kRows>(e, tile, position);
    } else {
        const uint32_t team = e.lay->team;
        RigidRun run;
        run.sm = e.sm; run.lay = e.lay; run.t = e.t; run.lane = e.lane; run.vstride = e.vstride;
        run.nheads = tile.nheads; run.nblocks = nb; run.tol = tile.tol;
#pragma unroll 1
        for (uint32_t k = 0u; k < count;) {
            const uint32_t b = order[k];
            if constexpr (NR > 0) { if (b == e.t->B) { descend_articulation<NR, kRows>(e, tile, position); ++k; continue; } }
            // the run of rigid blocks that share b's colour (a rigid block's 6 coordinates: one per lane)
            const uint32_t colour = blk_color(e, nb, b);
            uint32_t k_end = k + 1u;
#pragma unroll 1
            // colour 31 is the overflow colour (index_blocks hands it to every block past the 31st colour): not a set of
            // independent blocks, so they descend one by one
            while (colour < 31u && k_end < count && order[k_end] != e.t->B && blk_color(e, nb, order[k_end]) == colour) ++k_end;
            const bool shared_out = team > 1u && k_end - k > kBodyGroups && team_command(e.sm, *e.lay)->dead == 0u;
            const uint32_t stride = shared_out ? team : 1u;
            uint32_t seq = 0u;
            if (shared_out) {
                seq = team_post(e.sm, *e.lay, e.lane, kTeamDescend, k, k_end, position, tile);
#ifdef NKB_STAGE_TAPS
                if (e.cyc != nullptr && e.lane == 0u) e.cyc[31] += 1u;
#endif
            }
            RigidResult mine = {0.f, 0.f, 0u};
            bool collected = true;
            uint32_t share = 0u;
            // one pass takes the lead's share (all of the run when it is not shared out); further passes only run after a
            // helper failed to answer, and take the helpers' shares
#pragma unroll 1
            do {
                const RigidResult part = descend_share<NR>(run, k, k_end, share, stride, position);
                mine.momentum = fmaxf(mine.momentum, part.momentum); mine.residual = fmaxf(mine.residual, part.residual);
                mine.status |= part.status;
                if (shared_out && share == 0u) {
                    collected = team_collect(e.sm, *e.lay, e.lane, seq);
                    if (collected) {
#pragma unroll 1
                        for (uint32_t m = 1u; m < team; ++m) {
                            const float* r = team_result(e.sm, *e.lay, m);
                            mine.momentum = fmaxf(mine.momentum, r[0]); mine.residual = fmaxf(mine.residual, r[1]);
                            mine.status |= reinterpret_cast<const uint32_t*>(r)[2];
                        }
                    } else {
                        // a helper did not answer: flag the env, stop using the team, descend the helpers' shares here
                        mine.status |= kStatusTeamTimeout;
                        if (e.lane == 0u) team_command(e.sm, *e.lay)->dead = 1u;
                        __syncwarp();
                    }
                }
                ++share;
            } while (shared_out && !collected && share < team);
            tile.momentum = fmaxf(tile.momentum, mine.momentum);
            tile.residual = fmaxf(tile.residual, mine.residual);
            e.status |= mine.status;
            k = k_end;
        }
    }
}

struct DualMomentum { float t, beta; };

// Dual update over every head (block_descent_tile.cuh:2493-2595); returns the residual classes.
NKB_DEV void update_duals(Env& e, const Tile& tile, DualMomentum* mom, bool velocity, bool commit, float out[3]) {
    out[0] = out[1] = out[2] = 0.f;
    if (tile.nheads == 0u) return;
    float cn = 0.f, ct = 0.f, cj = 0.f;
    double restart = 0.0;
#pragma unroll 1
    for (uint32_t h = e.lane; h < tile.nheads; h += 32u) {
        const uint32_t fl = hu(e, HF_FLAGS, h);
        const bool contact = (fl & (kHeadContact | kHeadScalar)) == kHeadContact;
        const V3 tdual = commit ? hf3(e, HF_DUAL, h) : hf3(e, HF_BASE, h);
        const V3 res = hf3(e, HF_RES, h);
        const float rho = hf(e, HF_RHO, h), lower = hf(e, HF_LOWER, h), upper = hf(e, HF_UPPER, h), mu = hf(e, HF_MU, h);
        const float normal = scalar_impulse(tdual.x, rho, res.x, lower, upper).impulse;
        Relax rx;
        rx.step = hf3(e, HF_RXS, h); rx.weight = hf(e, HF_RXW, h); rx.point = hf3(e, HF_RXP, h);
        if (!commit) { rx.step = mk3(0.f, 0.f, 0.f); rx.weight = 0.f; rx.point = rx.step; }
        V3 dual;
        if (!contact) dual = mk3(normal, 0.f, 0.f);
        else {
            float iy, iz, c1, c2, c3;
            cone_impulse(tdual, rho, res.y, res.z, normal, mu, iy, iz, c1, c2, c3);
            dual = relax_contact_impulse_fast(tdual, mk3(normal, iy, iz), rx);
        }
        float sn, st;
        multiplier_steps_iso(tdual, dual, rho, contact ? mu : 0.f, sn, st);
        const V3 physical = commit ? dual : tdual;
        if (!contact) {
            const bool normal_row = (fl & kHeadContactNormal) != 0u;
            const float rate = -res.x;
            const float violation = physical.x > 0.f ? fabsf(rate) : fmaxf(-rate, 0.f);
            const float r = normal_row ? fmaxf(sn, violation) : sn;
            if (normal_row) cn = fmaxf(cn, residual_abs(r)); else cj = fmaxf(cj, residual_abs(r));
        } else {
            if (commit) { hst3(e, HF_RXS, h, rx.step); hf(e, HF_RXW, h) = rx.weight; hst3(e, HF_RXP, h, rx.point); }
            const V3 v = mk3(-res.x, -res.y, -res.z);
            cn = fmaxf(cn, residual_abs(physical.x > 0.f ? fabsf(v.x) : fmaxf(-v.x, 0.f)));
            ct = fmaxf(ct, residual_abs(fmaxf(st, fmaxf(along_axis(physical.y, v.y), along_axis(physical.z, v.z)))));
        }
        if (!commit) continue;
        if (velocity) set_head_lambda(e, h, dual);
        const V3 base = hf3(e, HF_BASE, h);
        restart += momentum_restart_iso(tdual, dual, base, rho, contact && mu > 0.f);
        if (mom != nullptr) hst3(e, HF_MOVE, h, base);
        hst3(e, HF_DUAL, h, dual);
        hst3(e, HF_BASE, h, dual);
    }
    __syncwarp();
    out[0] = warp_max(cn); out[1] = warp_max(ct); out[2] = warp_max(cj);
    if (mom != nullptr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) restart += __shfl_xor_sync(NKB_FULL, restart, o);
        if (restart > 0.0) mom->t = 1.0f;
        const float tn = 0.5f * (1.0f + sqrtf(fmaf(4.0f * mom->t, mom->t, 1.0f)));
        mom->beta = (mom->t - 1.0f) / tn;
        mom->t = tn;
#pragma unroll 1
        for (uint32_t h = e.lane; h < tile.nheads; h += 32u) {
            const bool contact = head_axes(e, h) == 3u;
            const float mu = hf(e, HF_MU, h);
            hst3(e, HF_DUAL, h, extrapolate_dual_iso(hf3(e, HF_MOVE, h), hf3(e, HF_BASE, h), mom->beta,
                                                     hf(e, HF_LOWER, h), hf(e, HF_UPPER, h), contact, mu));
        }
        __syncwarp();
    }
}

// Momentum balance of the free bodies, a group of lanes on each (BodyLanes): lane = row, the rows' Jacobian entries from the
// contact frames.
NKB_DEV void measure_bodies(Env& e, Tile& tile, bool reconstruct) {
    const TemplateView& t = *e.t;
    const BodyLanes g = body_lanes(e.lane);
    const uint32_t nb = tile.nblocks, row = g.j;
    const uint32_t* order = block_order(e, nb);
    const uint32_t blocks = order[nb];
    float worst = 0.f;
#pragma unroll 1
    for (uint32_t base = 0u; base < blocks; base += kBodyGroups) {
        const uint32_t turn = base + e.lane / kBodyLanes;
        const uint32_t b = turn < blocks ? order[turn] : t.B;
        const bool have = b != t.B;                                // the articulation's block has its own measure
        const uint32_t* inc = blk_inc(e, nb) + blk_inc_begin(e, nb, b);
        const uint32_t count = have ? blk_inc_begin(e, nb, b + 1u) - blk_inc_begin(e, nb, b) : 0u;
        double balance = 0.0;
        if (have) {
            const float* vel = block_vel(e, b, false);
            const float* fr = sm_bfree(e, b);
            if (row < 6u) {
                const float* bm = sm_bmass(e, b);
                if (row < 3u) balance = -(double)bm[0] * ((double)vel[row] - fr[row]);
                else {
                    const float m3 = row == 3u ? bm[1] : row == 4u ? bm[4] : bm[5], m4 = row == 3u ? bm[4] : row == 4u ? bm[2] : bm[6], m5 = row == 3u ? bm[5] : row == 4u ? bm[6] : bm[3];
                    balance = -((double)m3 * ((double)vel[3] - fr[3]) + (double)m4 * ((double)vel[4] - fr[4]) + (double)m5 * ((double)vel[5] - fr[5]));
                }
            }
#pragma unroll 1
            for (uint32_t k = 0u; k < count; ++k) {
                const uint32_t h = inc[k];
                const bool first_side = (hu(e, HF_OWNER, h) & 0xffffu) == b;
                const V3 w = body_row_axis(row, hf3(e, first_side ? HF_RA : HF_RB, h)), lam = head_lambda(e, h);
                const float sgn = first_side ? 1.f : -1.f;
                balance = fma((double)(sgn * dot(hf3(e, HF_N, h), w)), (double)lam.x, balance);
                balance = fma((double)(sgn * dot(hf3(e, HF_T1, h), w)), (double)lam.y, balance);
                balance = fma((double)(sgn * dot(hf3(e, HF_T2, h), w)), (double)lam.z, balance);
            }
        }
        __syncwarp();
        const bool finite = g.all(fabs(balance) <= FLT_MAX);
        float force[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) force[k] = __shfl_sync(NKB_FULL, (float)balance, g.first + k);
        if (have) {
            float residual = FLT_MAX;
            if (finite) {
                const float im = __ldg(t.inv_mass + b);
                const V3 ang = sym_mulv(sm_bwinv(e, b), mk3(force[3], force[4], force[5]));
                const float dir[6] = {force[0] * im, force[1] * im, force[2] * im, ang.x, ang.y, ang.z};
                residual = 0.f;
#pragma unroll
                for (int k = 0; k < 6; ++k) residual = fmaxf(residual, isfinite(dir[k]) ? fabsf(dir[k]) : FLT_MAX);
                if (reconstruct) {
                    if (g.j < 6u) block_vel(e, b, false)[g.j] += pick6(dir, g.j);
                    tile.momentum = fmaxf(tile.momentum, residual);
                }
            }
            worst = fmaxf(worst, residual);
        }
        __syncwarp();
    }
    tile.residual = fmaxf(tile.residual, warp_max_positive(worst));
    tile.momentum = warp_max(tile.momentum);
}

// Momentum balance of the articulation's block against the physical multipliers (block_descent_tile.cuh:2379-2489).
template <int NR>
NKB_DEV void measure_articulation(Env& e, Tile& tile, bool reconstruct) {
    const uint32_t nb = tile.nblocks, l = e.lane, b = e.t->B, dim = e.t->ndof;
    const uint32_t* inc = blk_inc(e, nb);
    if (dim == 0u) return;
    float* vel = block_vel(e, b, false);
    const float* fr = block_free(e, b);
    const uint32_t ib = blk_inc_begin(e, nb, b), ie = blk_inc_begin(e, nb, b + 1u);
    double balance[NR];
    bool coord[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) { balance[r] = 0.0; coord[r] = l + 32u * r < dim; }
    double* wide = reinterpret_cast<double*>(sm_vec(e, kVecS0));       // spans S0 and S1
#pragma unroll
    for (int r = 0; r < NR; ++r) wide[l + 32u * r] = coord[r] ? (double)vel[l + 32u * r] - fr[l + 32u * r] : 0.0;
    __syncwarp();
    {
        const uint32_t n4 = (dim + 3u) & ~3u;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const uint32_t c = l + 32u * r;
            if (!coord[r]) continue;
            balance[r] = (double)sm_fixed(e)[c] - mass_row_times(e, c, n4 >> 2, wide);
            if (tile.units)
#pragma unroll 1
                for (uint32_t slot = 0u; slot < 3u; ++slot) {
                    const uint32_t h = unit_table(e, nb)[slot * e.vstride + c];
                    if (h != kNoUnitHead) balance[r] += (double)hf(e, HF_UNITV, h) * hf(e, HF_LAMX, h);
                }
        }
#pragma unroll 1
        for (uint32_t k = ib; k < ie; ++k) {
            const uint32_t h = inc[k];
            const uint32_t jo = hu(e, HF_JOFF, h);
            if (jo & kUnitRow) continue;
            const V3 lam = head_lambda(e, h);
            const float* jr = sm_jpool(e) + jo;
            const bool cone = head_axes(e, h) == 3u;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const uint32_t c = l + 32u * r;
                if (!coord[r]) continue;
                balance[r] += (double)jr[c] * lam.x;
                if (cone) balance[r] += (double)jr[n4 + c] * lam.y + (double)jr[2u * n4 + c] * lam.z;
            }
        }
    }
    float force[NR], dir[NR];
    bool ok = true;
#pragma unroll
    for (int r = 0; r < NR; ++r) { force[r] = coord[r] ? (float)balance[r] : 0.f; dir[r] = 0.f; ok &= !coord[r] || fabs(balance[r]) <= FLT_MAX; }
    const bool finite = __all_sync(NKB_FULL, ok);
    float residual = FLT_MAX;
    if (finite) {
        solve_block_mass<NR>(e, b, force, dir);
        float worst = 0.f;
#pragma unroll
        for (int r = 0; r < NR; ++r) if (coord[r]) worst = fmaxf(worst, isfinite(dir[r]) ? fabsf(dir[r]) : FLT_MAX);
        residual = warp_max(worst);
    }
    tile.residual = fmaxf(tile.residual, residual);
    if (reconstruct && finite) {
#pragma unroll
        for (int r = 0; r < NR; ++r) if (coord[r]) vel[l + 32u * r] += dir[r];
        tile.momentum = fmaxf(tile.momentum, residual);
        __syncwarp();
    }
}

// Momentum balance of every moving block against the physical multipliers (block_descent_tile.cuh:2379-2489).
template <int NR, bool kRigid, bool kRows>
NKB_DEV void measure_primals(Env& e, Tile& tile, bool reconstruct) {
    if constexpr (kRigid) measure_bodies(e, tile, reconstruct);
    if constexpr (NR > 0) {
        measure_articulation<NR>(e, tile, reconstruct);
        if constexpr (kRows) {
            if (reconstruct && e.by_rows != 0u) {          // the velocity is the physical multipliers' now
                if (e.lane < e.rows) { const uint32_t entry = row_table(e)[e.lane]; row_y(e)[e.lane] = (double)comp(head_lambda(e, entry & 0xffffu), (int)(entry >> 16)); }
                __syncwarp();
            }
        }
    }
}

// The whole constraint solve of one env.  On entry the heads are built, the articulation's post-dynamics
// velocity is in (e.qd, sm_vel(root)) and free-body velocities are in sm_bvel.
// kRows: contacts can act on an articulation of more than 32 coordinates, so that its descent in the space of its rows is compiled in.
template <int NR, bool kRigid, bool kRows>
NKB_DEV void stage_solve(Env& e, uint32_t nheads) {
    const TemplateView& t = *e.t;
    const uint32_t l = e.lane, B = t.B, n = NR > 0 ? t.ndof : 0u;
    Tile tile;
    tile.nheads = nheads; tile.nblocks = B + (n != 0u ? 1u : 0u); tile.units = false;
    tile.momentum = tile.residual = 0.f; tile.tol = t.cfg.velocity_tolerance;
    // rigid blocks: free velocity, mass, carried constraint velocity (block_descent_rigid.cuh:4-48)
    if constexpr (kRigid)
#pragma unroll 1
    for (uint32_t b = l; b < B; b += 32u) {
        float* bv = sm_bvel(e, b);
        float* bf = sm_bfree(e, b);
        const float im = __ldg(t.inv_mass + b);
        uint32_t dim = 0u;
        if (im > 0.f && __ldg(t.body_to_link + b) == kNoLink) {
            const float* w = sm_bwinv(e, b);
            const double xx = w[0], yy = w[1], zz = w[2], xy = w[3], xz = w[4], yz = w[5];
            const double cxx = yy * zz - yz * yz, cyy = xx * zz - xz * xz, czz = xx * yy - xy * xy;
            const double cxy = xz * yz - xy * zz, cxz = xy * yz - xz * yy, cyz = xy * xz - xx * yz;
            const double det = xx * cxx + xy * cxy + xz * cxz;
            if (det > 0.0) {
                const double inv = 1.0 / det;
                float* bm = sm_bmass(e, b);
                bm[0] = (float)(1.0 / (double)im);
                bm[1] = (float)(cxx * inv); bm[2] = (float)(cyy * inv); bm[3] = (float)(czz * inv);
                bm[4] = (float)(cxy * inv); bm[5] = (float)(cxz * inv); bm[6] = (float)(cyz * inv);
                dim = 6u;
            } else e.status |= kStatusSolverFailure;
        }
        blk_dim(e, b) = dim;
        const float* carry = e.s->carry_rigid + ((size_t)e.env * B + b) * 6u;
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            bf[k] = bv[k];
            const float c = dim != 0u ? carry[k] : 0.f;
            bv[k] = bf[k] + (isfinite(c) ? c : 0.f);
        }
        float* ps = sm_bpseudo(e, b);
#pragma unroll
        for (int k = 0; k < 6; ++k) ps[k] = 0.f;
    }
    if (n != 0u && l == 0u) blk_dim(e, B) = n;
    // articulation coordinates: free = post-dynamics velocity
    if constexpr (NR > 0) {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const uint32_t at = l + 32u * r;
            const float qd_of_link = __shfl_sync(NKB_FULL, e.qd, e.dof_link[r]);
            if (at < n) {
                const float value = e.dof_comp[r] == kNoLink ? qd_of_link : sm_vel(e, e.dof_link[r])[e.dof_comp[r]];
                const float c = e.s->carry_artic[(size_t)e.env * n + at];
                sm_vec(e, kVecFree)[at] = value;
                sm_vec(e, kVecU)[at] = value + (isfinite(c) ? c : 0.f);
                sm_vec(e, kVecPseudo)[at] = 0.f;
            } else { sm_vec(e, kVecFree)[at] = 0.f; sm_vec(e, kVecU)[at] = 0.f; sm_vec(e, kVecPseudo)[at] = 0.f; }   // float4 readers see zeros past n
        }
    }
    __syncwarp();
    init_heads<NR, kRows>(e, tile, kRigid || nheads != 0u);
    tick(e, 8);
    float rows[3] = {0.f, 0.f, 0.f};
    float cls[4] = {0.f, 0.f, 0.f, 0.f};
    uint32_t sweeps = 0u, positions = 0u, pushes = 0u;
    DualMomentum mom = {1.0f, 0.0f};
    const uint32_t iterations = t.cfg.vel_iters;
    // One loop drives the velocity sweeps, the hand-over and the split-impulse position sweeps so that each of
    // the large pieces (block indexing, block descent, dual update, momentum balance) is instantiated once.
    // Without a row the articulation's velocity is the free one plus M^-1 times the drives' impulses: the momentum balance finds it
    // from the free velocity, and a second time from there, to make up for the factor's rounding.
    const bool linear = NR > 0 && !kRigid && nheads == 0u && iterations != 0u;
    if (linear)
#pragma unroll
        for (int r = 0; r < NR; ++r) sm_vec(e, kVecU)[l + 32u * r] = sm_vec(e, kVecFree)[l + 32u * r];
    __syncwarp();
    enum { kPhaseVelocity, kPhaseHandOver, kPhasePosition, kPhaseDone };
    int phase = kPhaseVelocity;
    bool reindex = true;
#pragma unroll 1
    while (phase != kPhaseDone) {
        if (reindex) {
            index_blocks<kRigid>(e, tile, phase == kPhaseVelocity);
            reindex = false;
            if (phase == kPhaseVelocity) { init_residuals(e, tile); tick(e, 9); if (iterations == 0u) phase = kPhaseHandOver; }
        }
        if (phase == kPhaseHandOver) {
            if (l < 4u) e.s->solver_residual[(size_t)e.env * 4u + l] = cls[l];
            if (l == 0u) e.s->solver_sweeps[e.env] = sweeps;
            // velocities back to the links, carried velocities to global memory
            if (n != 0u) {
                const float* U = sm_vec(e, kVecU);
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const uint32_t at = l + 32u * r;
                    if (at < n) {
                        e.s->carry_artic[(size_t)e.env * n + at] = U[at] - sm_vec(e, kVecFree)[at];
                        if (e.dof_comp[r] != kNoLink) sm_vel(e, e.dof_link[r])[e.dof_comp[r]] = U[at];
                    }
                }
                if (l < t.L && joint_dofs(e.jtype) == 1u) e.qd = U[e.link_dof];
            }
            if constexpr (kRigid)
#pragma unroll 1
            for (uint32_t b = l; b < B; b += 32u) {
                float* carry = e.s->carry_rigid + ((size_t)e.env * B + b) * 6u;
                const float* bv = sm_bvel(e, b);
                const float* bf = sm_bfree(e, b);
#pragma unroll
                for (int k = 0; k < 6; ++k) carry[k] = blk_dim(e, b) != 0u ? bv[k] - bf[k] : 0.f;
            }
            __syncwarp();
            phase = kPhaseDone;
            // split-impulse position pass: every head becomes a scalar push-out row (ops/block_descent.cu:1734-1753)
            if (t.cfg.pos_iters != 0u && nheads != 0u) {
                bool push = false, coupled = false;
#pragma unroll 1
                for (uint32_t h = l; h < nheads; h += 32u) {
                    const uint32_t fl = hu(e, HF_FLAGS, h);
                    const bool spec = (fl & kHeadSpeculative) != 0u;
                    const float slop = spec ? 0.f : t.cfg.pos_slop;
                    const float pen_row = hf(e, HF_PEN, h);
                    const bool active = (fl & kHeadVelocityOnly) == 0u && (spec || pen_row > slop || hf(e, HF_DUAL, h) != 0.f);
                    float bias = 0.f, rounding = 0.f;
                    if (active) {
                        const float penetration = fmaxf(pen_row - slop, 0.f);
                        if (spec) {
                            const float cd = sm_cdepth(e)[hu(e, HF_REF, h) & 0xffffu];
                            const double depth = (double)cd - slop, reserve = (double)pen_row - cd;
                            const double correction = t.cfg.pos_beta * fmax(depth, 0.0) + reserve;
                            const double target = fmin(depth, 0.0) + correction;
                            double velocity = 0.0;
#pragma unroll 1
                            for (uint32_t side = 0u; side < 2u; ++side) {
                                const uint32_t b = head_owner(e, h, side);
                                if (b == kNoBlock16) continue;
                                velocity += (double)head_row_dot(e, h, side, 0u, b, block_vel(e, b, false));
                            }
                            const double limit = fmin(correction / t.cfg.dt, (double)t.cfg.baumgarte_max_velocity);
                            bias = (float)fmin(target / t.cfg.dt - velocity, limit);
                            rounding = (float)(target > 0.0 ? 0.0 : fmax(reserve, 0.0) / t.cfg.dt);
                        } else {
                            bias = fminf(t.cfg.pos_beta * penetration / t.cfg.dt, t.cfg.baumgarte_max_velocity);
                        }
                    } else hu(e, HF_OWNER, h) = kNoBlock16 | (kNoBlock16 << 16);
                    const uint32_t o = hu(e, HF_OWNER, h);
                    coupled |= (o & 0xffffu) != kNoBlock16 && (o >> 16) != kNoBlock16;
                    hu(e, HF_FLAGS, h) = fl | kHeadScalar;
                    hf(e, HF_LOWER, h) = 0.f; hf(e, HF_UPPER, h) = FLT_MAX;
                    hf(e, HF_MU, h) = 0.f;
                    hst3(e, HF_RES, h, mk3(bias, 0.f, 0.f));
                    hst3(e, HF_DUAL, h, mk3(0.f, 0.f, 0.f));
                    push |= bias > rounding;
                }
                push = __any_sync(NKB_FULL, push); coupled = __any_sync(NKB_FULL, coupled);
                __syncwarp();
                if (push) {
                    if (NR > 0 && e.by_rows != 0u) { if (l < e.rows) row_y(e)[l] = 0.0; __syncwarp(); }
                    phase = kPhasePosition; reindex = true; positions = coupled ? t.cfg.pos_iters : 1u; pushes = 0u; }
            }
            continue;
        }
        if (phase == kPhaseVelocity) { ++sweeps; tile.momentum = 0.f; tile.residual = 0.f; }
        if (!linear) descend_blocks<NR, kRigid, kRows>(e, tile, phase == kPhasePosition);
        if (phase == kPhasePosition) {
            if (++pushes >= positions) { phase = kPhaseDone; continue; }
        } else tick(e, 10);
        update_duals(e, tile, phase == kPhaseVelocity ? &mom : nullptr, phase == kPhaseVelocity, true, rows);
        if (phase == kPhasePosition) continue;
        tick(e, 24);
        // momentum balance: plain measure, reconstruction when only the primal lags, re-measure after it
#pragma unroll 1
        for (int stage = 0; stage < 3; ++stage) {
            const float worst_row = fmaxf(fmaxf(rows[0], rows[1]), rows[2]);
            bool run = true;
            if (linear) {}
            else if (stage == 0) run = sweeps == iterations || fmaxf(worst_row, tile.residual) < tile.tol;
            else if (stage == 1) run = worst_row < tile.tol && tile.residual >= tile.tol && tile.residual < FLT_MAX;
            if (stage == 1 && !run) break;
            const bool reconstruct = stage == 1 || (linear && stage == 0);
            if (run) { measure_primals<NR, kRigid, kRows>(e, tile, reconstruct); tick(e, 25); tick_count(e, 27); }
            if (linear && !(tile.residual < FLT_MAX)) { e.status |= kStatusSolverFailure; break; }
            if (reconstruct) {
                if (!(tile.residual < FLT_MAX)) break;
                init_residuals(e, tile);
                update_duals(e, tile, nullptr, true, false, rows);
                tile.residual = 0.f;
                tick(e, 26);
            }
        }
        cls[0] = rows[0]; cls[1] = rows[1]; cls[2] = rows[2]; cls[3] = tile.residual;
        const float largest = fmaxf(fmaxf(rows[0], rows[1]), fmaxf(rows[2], tile.residual));
        tick(e, 11);
        if (sweeps >= iterations || largest < tile.tol || largest == FLT_MAX) phase = kPhaseHandOver;
    }
    tick(e, 14);
    if (e.s->dbg_qdot_pseudo != nullptr) for (uint32_t at = l; at < n; at += 32u) e.s->dbg_qdot_pseudo[(size_t)e.env * n + at] = sm_vec(e, kVecPseudo)[at];
}

}  // namespace nkb
