// The articulation's descent in the space of its constraint rows.
//
// At a block's minimum M (u - u_free) = f_fixed + J^T f(u), so u = u_b + M^-1 J^T y with u_b = u_free + M^-1 f_fixed and y = f: the
// unknowns are the m multipliers y of the rows that act on the articulation, not its n coordinates.  With W = J M^-1 J^T a Newton
// step of the block's problem, H d = J^T (f - y) with H = M + J^T C J, is d = M^-1 J^T dy with (1 + C W) dy = f - y; the rows move
// by W dy, the line's slope at step a is sum (y + a dy - f(a)) (W dy), its curvature dy^T W dy + (W dy)^T C (W dy).  Nothing inside
// the loop is as wide as the articulation: a humanoid on two feet has 6 rows and 35 coordinates, and a contact between
// two limbs adds three rows instead of joining branches of the tree.  C = R R^T with one column of R per row that responds (a
// sliding contact has one for both tangents), and dy = (f - y) + R w with (1 + R^T W R) w = - R^T W (f - y): symmetric, every
// pivot at least 1, and only as wide as the rows that respond.
//
// M^-1 J^T and W are built once a step from the mass matrix's factor, a lane to a row (build_rows); W's diagonal is also the rows'
// response that the penalties want.  Envs with more rows than solve_rows holds (row_cap), or a response below zero, take the descents in coordinates.
//
// It is taken by articulations of more than 32 coordinates: 2048 humanoids, 4 steps, 1.97 ms (in coordinates 3.50).  Up to 32 the descent in
// coordinates stays: a quadruped's 18 make a system about as cheap as W, and an env at rest, one Newton step to a descent, would pay for building
// W (4096 standing quadrupeds 198 us against 183).
// What bounds it is the chain of one warp: build_rows over the joints, one after another, solve_rows over groups of three rows, the line search.
#pragma once
#include "nkb_laws.cuh"
#include "nkb_rows.cuh"

namespace nkb {

// Where a row's penalty times its response passes this, the envs descend in coordinates: contacts that lock a limb (three on eight joints) leave
// W without rank, 32-bit pivots of 1 + R^T W R lose the 1 beside entries of 1e6 and more, and the descent ends nowhere (7.8 rad/s off in one
// env of 96; 8e-5 with the line here, 1.7e-4 in coordinates).  A quadruped's rows stay below 1e3.  A descent that runs out of steps all the
// same goes on in coordinates too.
constexpr float kRowStiffness = 1.0e4f;

NKB_DEV float* row_x(const Env& e) { return e.sm + e.lay->chol; }                                               // M^-1 J^T by row; last M^-1 times the drives
NKB_DEV float* row_w(const Env& e) { return row_x(e) + (e.t->row_cap + 1u) * e.t->row_stride; }               // J M^-1 J^T, rows of row_words words
NKB_DEV uint32_t row_words(const Env& e) { return e.t->row_cap | 1u; }
NKB_DEV uint32_t* row_table(const Env& e) { return reinterpret_cast<uint32_t*>(row_w(e) + e.t->row_cap * row_words(e)); }      // head | axis << 16
// The rows' multipliers.  In 64 bits: the rows are stiff, so an impulse rounded to 32 bits (1.5e-8 of 0.25 N s) moves a light joint by 1.5e-6
// rad/s, while the rounding of a row's response is divided by 1 + C W.
NKB_DEV double* row_y(const Env& e) { return reinterpret_cast<double*>(row_x(e) + row_space_head(e.t->row_cap, e.t->row_stride)); }

// J_r . v over the articulation's coordinates, v in shared memory with zeros past the last one; in 64 bits, since what a row moves by is
// a small difference of large terms.
NKB_DEV double row_dot(const Env& e, uint32_t h, uint32_t axis, const double* v) {
    const uint32_t jo = hu(e, HF_JOFF, h), chunks = (e.t->ndof + 3u) >> 2;
    if (jo & kUnitRow) return (double)hf(e, HF_UNITV, h) * v[jo & 0xffffu];
    const float4* j4 = reinterpret_cast<const float4*>(sm_jpool(e) + jo) + axis * chunks;
    const double2* v2 = reinterpret_cast<const double2*>(v);
    double s0 = 0.0, s1 = 0.0;
#pragma unroll 1
    for (uint32_t c = 0u; c < chunks; ++c) {
        const float4 a = j4[c];
        const double2 p = v2[2u * c], q = v2[2u * c + 1u];
        s0 = fma((double)a.x, p.x, s0); s1 = fma((double)a.y, p.y, s1); s0 = fma((double)a.z, q.x, s0); s1 = fma((double)a.w, q.y, s1);
    }
    return s0 + s1;
}

// Numbers the rows that act on the articulation (three per contact head, then one per joint row), solves M x = J^T for each and
// for the drives' impulses, and multiplies out W.  False where there are more rows than the slice holds, or a response is below zero.
// A lane walks the tree for its row: joints from the last to the first push their share to the base and to their ancestors, then
// the base's 6 x 6, then joints from the first to the last; the factor's rows are read by all lanes at once.
template <int NR>
NKB_DEV bool build_rows(Env& e, uint32_t nheads) {
    const TemplateView& t = *e.t;
    const uint32_t l = e.lane, n = t.ndof, xs = t.row_stride, chunks = (n + 3u) >> 2;
    uint32_t* table = row_table(e);
    uint32_t contacts = 0u, units = 0u;
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
        uint32_t at = 0u, unit_at = 3u * contacts;
#pragma unroll 1
        for (uint32_t base = 0u; base < nheads; base += 32u) {
            const uint32_t h = base + l;
            bool mine = false, unit = false;
            if (h < nheads) {
                const uint32_t o = hu(e, HF_OWNER, h);
                mine = (o & 0xffffu) == t.B || (o >> 16) == t.B;
                unit = (hu(e, HF_JOFF, h) & kUnitRow) != 0u;
            }
            const uint32_t mc = __ballot_sync(NKB_FULL, mine && !unit), mu = __ballot_sync(NKB_FULL, mine && unit), below = (1u << l) - 1u;
            if (pass != 0 && mine) {
                if (unit) table[unit_at + __popc(mu & below)] = h;
                else {
                    const uint32_t r = at + 3u * __popc(mc & below);
                    table[r] = h; table[r + 1u] = h | 0x10000u; table[r + 2u] = h | 0x20000u;
                }
            }
            at += 3u * __popc(mc); unit_at += __popc(mu);
            if (pass == 0) { contacts += __popc(mc); units += __popc(mu); }
        }
        if (pass == 0 && 3u * contacts + units > t.row_cap) return false;
    }
    const uint32_t m = 3u * contacts + units;
    e.rows = m;
    __syncwarp();
    float* X = row_x(e);
#pragma unroll 1
    for (uint32_t k = l; k < (m + 1u) * chunks; k += 32u) {
        const uint32_t r = k / chunks, c = 4u * (k - r * chunks);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r == m) {
            const float* f = sm_fixed(e);
            v.x = f[c]; v.y = c + 1u < n ? f[c + 1u] : 0.f; v.z = c + 2u < n ? f[c + 2u] : 0.f; v.w = c + 3u < n ? f[c + 3u] : 0.f;
        } else {
            const uint32_t entry = table[r], h = entry & 0xffffu, jo = hu(e, HF_JOFF, h);
            if (jo & kUnitRow) {
                const uint32_t at = (jo & 0xffffu) - c;
                const float unit = hf(e, HF_UNITV, h);
                v = make_float4(at == 0u ? unit : 0.f, at == 1u ? unit : 0.f, at == 2u ? unit : 0.f, at == 3u ? unit : 0.f);
            } else v = reinterpret_cast<const float4*>(sm_jpool(e) + jo)[(entry >> 16) * chunks + (c >> 2)];
        }
        *reinterpret_cast<float4*>(X + r * xs + c) = v;
    }
    __syncwarp();
    const float* factor = sm_factor(e);
    const uint32_t stride = t.tree_stride, first = tree_first<NR>(e), start = t.floating_root ? 6u : 0u;
    const bool live = l <= m;
    float* x = X + (live ? l : 0u) * xs;
    float z[kTreeBase];
#pragma unroll
    for (int k = 0; k < kTreeBase; ++k) z[k] = t.floating_root ? x[k] : 0.f;
    __syncwarp();
#pragma unroll 1
    for (uint32_t c = n; c-- > start;) {
        const float* src = factor + ((c & 31u) - first) * stride;
        const float y = live ? x[c] * src[7] : 0.f;
        if (!__any_sync(NKB_FULL, y != 0.f)) continue;
        const float4 b0 = reinterpret_cast<const float4*>(src)[0];
        const float2 b1 = reinterpret_cast<const float2*>(src)[2];
        z[0] = fmaf(-b0.x, y, z[0]); z[1] = fmaf(-b0.y, y, z[1]); z[2] = fmaf(-b0.z, y, z[2]);
        z[3] = fmaf(-b0.w, y, z[3]); z[4] = fmaf(-b1.x, y, z[4]); z[5] = fmaf(-b1.y, y, z[5]);
        const uint32_t* lane = t.tree_lanes + (c & 31u) * kTreeLaneWords;
        const uint32_t level = (__ldg(lane) >> 8) & 0xffu;
        if (live) {
            x[c] = y;
#pragma unroll 1
            for (uint32_t p = 0u; p < level; ++p) {
                const uint32_t a = (__ldg(lane + 2 + (p >> 2)) >> (8u * (p & 3u))) & 0xffu;
                x[a] = fmaf(-src[8u + p], y, x[a]);
            }
        }
    }
    float s[kTreeBase];
#pragma unroll
    for (int k = 0; k < kTreeBase; ++k) s[k] = 0.f;
    if (t.floating_root) {
        const float* block = factor + tree_rows<NR>(e) * stride + 48;
        float a[28];
#pragma unroll
        for (int k = 0; k < 7; ++k) { const float4 v = reinterpret_cast<const float4*>(block)[k]; a[4 * k] = v.x; a[4 * k + 1] = v.y; a[4 * k + 2] = v.z; a[4 * k + 3] = v.w; }
#pragma unroll
        for (int k = 0; k < kTreeBase; ++k) {
            z[k] *= a[21 + k];
#pragma unroll
            for (int i = k + 1; i < kTreeBase; ++i) z[i] = fmaf(-a[i * (i + 1) / 2 + k], z[k], z[i]);
        }
#pragma unroll
        for (int k = kTreeBase - 1; k >= 0; --k) {
            s[k] = z[k] * a[21 + k];
#pragma unroll
            for (int i = 0; i < k; ++i) z[i] = fmaf(-a[k * (k + 1) / 2 + i], s[k], z[i]);
        }
        if (live) {
            reinterpret_cast<float2*>(x)[0] = make_float2(s[0], s[1]); reinterpret_cast<float2*>(x)[1] = make_float2(s[2], s[3]);
            reinterpret_cast<float2*>(x)[2] = make_float2(s[4], s[5]);
        }
    }
    if (live)
#pragma unroll 1
        for (uint32_t c = start; c < n; ++c) {
            const float* src = factor + ((c & 31u) - first) * stride;
            const uint32_t* lane = t.tree_lanes + (c & 31u) * kTreeLaneWords;
            const uint32_t level = (__ldg(lane) >> 8) & 0xffu;
            const float4 b0 = reinterpret_cast<const float4*>(src)[0];
            const float4 b1 = reinterpret_cast<const float4*>(src)[1];
            float g = fmaf(-b0.x, s[0], x[c]), q = -b0.y * s[1];
            g = fmaf(-b0.z, s[2], g); q = fmaf(-b0.w, s[3], q); g = fmaf(-b1.x, s[4], g); q = fmaf(-b1.y, s[5], q);
#pragma unroll 1
            for (uint32_t p = 0u; p < level; ++p) {
                const uint32_t a = (__ldg(lane + 2 + (p >> 2)) >> (8u * (p & 3u))) & 0xffu;
                g = fmaf(-src[8u + p], x[a], g);
            }
            x[c] = (g + q) * b1.w;
        }
    __syncwarp();
    // W, lane = row: J_l X_j, three j at a time (a contact's rows)
    const uint32_t entry = l < m ? table[l] : 0u, h = entry & 0xffffu;
    const float* diagonal = row_w(e) + l * (row_words(e) + 1u);
    if (l < m) {
        const uint32_t jo = hu(e, HF_JOFF, h), at = jo & 0xffffu;
        const bool unit = (jo & kUnitRow) != 0u;
        const float4* j4 = reinterpret_cast<const float4*>(sm_jpool(e) + (unit ? 0u : jo)) + (entry >> 16) * chunks;
        const float value = unit ? hf(e, HF_UNITV, h) : 0.f;
        float* mine = row_w(e) + l * row_words(e);
#pragma unroll 1
        for (uint32_t j = 0u; j < m; j += 3u) {
            const uint32_t step1 = j + 1u < m ? xs : 0u, step2 = j + 2u < m ? step1 + xs : step1;
            const float* x0 = X + j * xs;
            float s0 = 0.f, s1 = 0.f, s2 = 0.f;
            if (unit) { s0 = value * x0[at]; s1 = value * x0[step1 + at]; s2 = value * x0[step2 + at]; }
            else
#pragma unroll 1
                for (uint32_t c = 0u; c < chunks; ++c) {
                    const float4 v = j4[c], p = reinterpret_cast<const float4*>(x0)[c], q = reinterpret_cast<const float4*>(x0 + step1)[c], w = reinterpret_cast<const float4*>(x0 + step2)[c];
                    s0 = fmaf(v.x, p.x, s0); s1 = fmaf(v.x, q.x, s1); s2 = fmaf(v.x, w.x, s2);
                    s0 = fmaf(v.y, p.y, s0); s1 = fmaf(v.y, q.y, s1); s2 = fmaf(v.y, w.y, s2);
                    s0 = fmaf(v.z, p.z, s0); s1 = fmaf(v.z, q.z, s1); s2 = fmaf(v.z, w.z, s2);
                    s0 = fmaf(v.w, p.w, s0); s1 = fmaf(v.w, q.w, s1); s2 = fmaf(v.w, w.w, s2);
                }
            mine[j] = s0;
            if (j + 1u < m) mine[j + 1u] = s1;
            if (j + 2u < m) mine[j + 2u] = s2;
        }
        row_y(e)[l] = 0.0;
    }
    // W's diagonal is a sum of both signs: a response that rounds below zero, which init_heads takes for a failure, is one for the coordinates
    if (__any_sync(NKB_FULL, l < m && !(*diagonal >= 0.f))) return false;
    if (l < m && (entry >> 16) == 0u) hf(e, HF_RHO, h) = *diagonal;          // the response of the head's normal row (init_heads)
    __syncwarp();
    return true;
}

// W v, lane = row
NKB_DEV float row_product(const Env& e, uint32_t m, float v) {
    const float* mine = row_w(e) + min(e.lane, m - 1u) * row_words(e);
    float s0 = 0.f, s1 = 0.f, s2 = 0.f;
#pragma unroll 1
    for (uint32_t j = 0u; j < m; j += 3u) {             // lanes past the last row carry zeros, their columns are the last row's
        s0 = fmaf(mine[j], __shfl_sync(NKB_FULL, v, j), s0);
        s1 = fmaf(mine[min(j + 1u, m - 1u)], __shfl_sync(NKB_FULL, v, j + 1u), s1);
        s2 = fmaf(mine[min(j + 2u, m - 1u)], __shfl_sync(NKB_FULL, v, j + 2u), s2);
    }
    return s0 + (s1 + s2);
}
// X v, lane = coordinate lane + 32 r
template <int NR>
NKB_DEV void row_spread(const Env& e, uint32_t m, double v, double (&out)[NR]) {
    const float* X = row_x(e) + e.lane;
    const uint32_t n = e.t->ndof;
#pragma unroll 1
    for (uint32_t j = 0u; j < m; ++j, X += e.t->row_stride) {
        const double vj = __shfl_sync(NKB_FULL, v, j);
#pragma unroll
        for (int r = 0; r < NR; ++r) if (e.lane + 32u * r < n) out[r] = fma((double)X[32 * r], vj, out[r]);
    }
}

// What a lane knows of its row for a descent.
struct RowLane {
    bool live, tangent;
    uint32_t partner;                   // the other tangent's lane
    float dual, rho, res, lower, upper, radius;
};
struct RowResponse { float impulse, curvature, cross; };         // curvature of the row, and against its partner
// The row laws (scalar_impulse, cone_impulse) with a lane to a row.
NKB_DEV RowResponse row_respond(const RowLane& a, float move) {
    const float residual = a.res - move;
    float q = fmaf(a.rho, residual, a.dual);
    if (a.tangent) q = cone_argument_unit(a.dual, a.rho, residual);
    const float other = __shfl_sync(NKB_FULL, q, a.partner);
    RowResponse out = {0.f, 0.f, 0.f};
    if (!a.live || a.rho <= 0.0f) return out;
    if (!a.tangent) {
        out.impulse = q < a.lower ? a.lower : (q > a.upper ? a.upper : q);
        out.curvature = q != q ? q : (a.lower < a.upper && q >= a.lower && q <= a.upper ? a.rho : 0.0f);
    } else if (a.radius != 0.f) {
        const float n2 = fmaf(q, q, __fmul_rn(other, other)), m2 = fmaf(other, other, __fmul_rn(q, q));       // the pair decides alike
        if (fminf(n2, m2) <= a.radius * a.radius) { out.impulse = q; out.curvature = a.rho; }
        else {
            const float inv = rsqrtf(fminf(n2, m2));
            const float own = q * inv, off = other * inv, cs = a.rho * a.radius * inv;
            out.impulse = a.radius * own;
            out.curvature = cs * off * off; out.cross = -(cs * own * off);
        }
    }
    return out;
}

// w with (1 + R^T W R) w = - R^T W r, and from it dy = r + R w; s = W r.  `ra` is the entry of R's column on the lane's own row, `rb` the one
// on its partner's.  Block Gauss-Jordan over the groups of three rows in which one responds, lane = row: a lane holds its row over
// the groups ahead; the group at hand is inverted by every lane for itself, and the rows of the others come by symmetry, from the lanes
// of their columns.  Every row is reduced, so the right-hand side ends as the solution.
template <int kRowGroups>
NKB_DEV bool solve_rows(const Env& e, uint32_t m, uint32_t partner, float ra, float rb, float r, float s, float& dy) {
    const uint32_t l = e.lane, active = __ballot_sync(NKB_FULL, ra != 0.f || rb != 0.f), slides = __ballot_sync(NKB_FULL, rb != 0.f);
    const uint32_t last = m - 1u, own = min(l, last) * row_words(e), beside = min(l + 1u, last) * row_words(e);
    const float* W = row_w(e);
    const uint32_t firsts = (active | (active >> 1) | (active >> 2)) & 0x09249249u;            // groups with a row that responds, by their first lane
    float b = -(ra * s);
    if (slides != 0u) b = fmaf(-rb, __shfl_sync(NKB_FULL, s, partner), b);
    // this lane's row of the matrix
    float a[3 * kRowGroups];
    uint32_t todo = firsts;
#pragma unroll
    for (int g = 0; g < kRowGroups; ++g) {
        if (todo == 0u) break;
        const uint32_t c = (uint32_t)__ffs(todo) - 1u;
        todo &= todo - 1u;
        const uint32_t c1 = min(c + 1u, last), c2 = min(c + 2u, last);
        float w0 = ra * W[own + c], w1 = ra * W[own + c1], w2 = ra * W[own + c2];
        if (slides != 0u) { w0 = fmaf(rb, W[beside + c], w0); w1 = fmaf(rb, W[beside + c1], w1); w2 = fmaf(rb, W[beside + c2], w2); }
        const float r0 = __shfl_sync(NKB_FULL, ra, c), r1 = __shfl_sync(NKB_FULL, ra, c + 1u), r2 = __shfl_sync(NKB_FULL, ra, c + 2u);
        a[3 * g] = fmaf(w0, r0, l == c ? 1.f : 0.f);
        a[3 * g + 1] = fmaf(w1, r1, l == c + 1u ? 1.f : 0.f);
        a[3 * g + 2] = fmaf(w2, r2, l == c + 2u ? 1.f : 0.f);
        if (slides != 0u) a[3 * g + 1] = fmaf(w2, __shfl_sync(NKB_FULL, rb, c + 1u), a[3 * g + 1]);        // a slide's column lies with the first tangent
    }
    bool valid = true;
#pragma unroll 1
    for (uint32_t left = firsts; left != 0u; left &= left - 1u) {
        const uint32_t c = (uint32_t)__ffs(left) - 1u, place = l - c;
        const float p00 = __shfl_sync(NKB_FULL, a[0], c), p10 = __shfl_sync(NKB_FULL, a[0], c + 1u), p20 = __shfl_sync(NKB_FULL, a[0], c + 2u);
        const float p11 = __shfl_sync(NKB_FULL, a[1], c + 1u), p21 = __shfl_sync(NKB_FULL, a[1], c + 2u), p22 = __shfl_sync(NKB_FULL, a[2], c + 2u);
        const float b0 = __shfl_sync(NKB_FULL, b, c), b1 = __shfl_sync(NKB_FULL, b, c + 1u), b2 = __shfl_sync(NKB_FULL, b, c + 2u);
        const float i0 = __fdividef(1.f, p00), l1 = p10 * i0, l2 = p20 * i0, d1 = fmaf(-l1, p10, p11), i1 = __fdividef(1.f, d1);
        const float o = fmaf(-l2, p10, p21), l3 = o * i1, d2 = fmaf(-l3, o, fmaf(-l2, p20, p22)), i2 = __fdividef(1.f, d2);
        valid &= pivot_valid(p00) && pivot_valid(d1) && pivot_valid(d2);
        // the multiples of the group's rows that this row gives up: its entries times the block's inverse; in the group itself what the inverse leaves of its own row
        const float e0 = place == 0u ? 1.f : 0.f, e1 = place == 1u ? 1.f : 0.f, e2 = place == 2u ? 1.f : 0.f;
        const bool inside = place < 3u;
        const float v0 = inside ? e0 : a[0], v1 = fmaf(-l1, v0, inside ? e1 : a[1]), v2 = fmaf(-l3, v1, fmaf(-l2, v0, inside ? e2 : a[2]));
        float t2 = v2 * i2, t1 = fmaf(-l3, t2, v1 * i1), t0 = fmaf(-l1, t1, fmaf(-l2, t2, v0 * i0));
        if (inside) { t0 = e0 - t0; t1 = e1 - t1; t2 = e2 - t2; }
        b = fmaf(-t0, b0, b); b = fmaf(-t1, b1, b); b = fmaf(-t2, b2, b);
        const float a0 = a[0], a1 = a[1], a2 = a[2];
        uint32_t ahead = left & (left - 1u);
#pragma unroll
        for (int g = 1; g < kRowGroups; ++g) {
            if (ahead == 0u) break;
            const uint32_t k = (uint32_t)__ffs(ahead) - 1u;
            ahead &= ahead - 1u;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                float v = a[3 * g + q];
                v = fmaf(-t0, __shfl_sync(NKB_FULL, a0, k + q), v);
                v = fmaf(-t1, __shfl_sync(NKB_FULL, a1, k + q), v);
                a[3 * (g - 1) + q] = fmaf(-t2, __shfl_sync(NKB_FULL, a2, k + q), v);
            }
        }
    }
    dy = fmaf(ra, b, r);
    if (slides != 0u) dy += __shfl_sync(NKB_FULL, rb * b, partner);
    return valid;
}

}  // namespace nkb
