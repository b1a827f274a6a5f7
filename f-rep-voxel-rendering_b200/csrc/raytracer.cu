// Raytracer kernel (sm_100a): one thread per pixel.
//
// Replaces vulkan/shaders/raytracer/main.comp (+ tape/gradient.comp,
// random.comp) and Raytracer::Trace (vulkan/src/engine/raytracer.cpp:243-272):
// ray generation, kd-restart DDA through the multi-level tree, forward-mode
// gradient of the hit node's tape for the normal, diffuse + ambient shading,
// optional shadow rays, rgba8 (and hit records) into device buffers.
//
// Blocks are 8 x 8 pixel tiles, so that neighbouring rays (which walk the same
// nodes and usually share the hit node's tape) sit in the same warp.
#include <algorithm>
#include "cell_div.h"
#include "device_common.cuh"
#include "kernels.h"

namespace frep {
namespace dev {

constexpr uint32_t RENDER_THREADS = 64;

struct RHit {
    float t;
    uint32_t node, level, cell, steps;
};

// What a step needs of a level, in a warp's shared memory (two 16-byte reads
// where a ray changes its level): the address of the level's first record and
// the bytes of one, the words of a mask, the cells along an axis, the cell size
// and its reciprocal, and the largest distance that div_by takes (0: none).
struct __align__(16) Level {
    const uint32_t* nodes;
    uint32_t size, words;
    float dim, cell, rcell, vmax;
};

template <bool CMP>
__device__ __forceinline__ void load_levels(const RenderArgs& A, Level* lv) {
    const uint32_t l = threadIdx.x & 31;
    if (l < A.levels) {
        const unsigned long long ofs = CMP ? A.node_ofs[l] : __ldg(&A.hdr->node_ofs[l]);
        const uint32_t dim = A.dims[l];
        const float cs = A.cell_size[l];
        lv[l] = Level{A.nodes + ofs, A.node_size[l] * 4, dim * dim * dim >> 5, (float)dim, cs, __frcp_rn(cs),
                      cs >= DIV_BY_DMIN && cs <= DIV_BY_DMAX ? DIV_BY_MAX : 0.0f};
    }
    __syncwarp();
}

__device__ __forceinline__ const uint32_t* node_rec(const Level& l, uint32_t node) {
    return reinterpret_cast<const uint32_t*>(reinterpret_cast<const char*>(l.nodes) +
                                             (unsigned long long)node * l.size);
}

// Where a node record keeps its masks and children. CMP = false: the
// reference's layout (node.comp:4-72), [tape, coords, leaf, interior,
// childList[dim^3]]; CMP = true: the compact layout, [tape, leaf[W],
// interior[W], prefix[W], base] (last level [tape, leaf[W]]), W = dim^3 / 32,
// whose interior children are numbered consecutively from `base` in cell
// order, prefix[w] = interior cells before word w.
template <bool CMP>
struct Layout;
template <>
struct Layout<false> {
    static __device__ __forceinline__ uint32_t leaf_word(const uint32_t* r, uint32_t W, uint32_t idx) {
        return __ldg(&r[4 + (idx >> 5)]);
    }
    static __device__ __forceinline__ uint32_t interior_word(const uint32_t* r, uint32_t W, uint32_t idx) {
        return __ldg(&r[4 + W + (idx >> 5)]);
    }
    // The child node of an interior cell, whose interior word is iw.
    static __device__ __forceinline__ uint32_t child(const uint32_t* r, uint32_t W, uint32_t idx, uint32_t iw) {
        return __ldg(&r[4 + 2 * W + idx]);
    }
};
template <>
struct Layout<true> {
    static __device__ __forceinline__ uint32_t leaf_word(const uint32_t* r, uint32_t W, uint32_t idx) {
        return __ldg(&r[1 + (idx >> 5)]);
    }
    static __device__ __forceinline__ uint32_t interior_word(const uint32_t* r, uint32_t W, uint32_t idx) {
        return __ldg(&r[1 + W + (idx >> 5)]);
    }
    static __device__ __forceinline__ uint32_t child(const uint32_t* r, uint32_t W, uint32_t idx, uint32_t iw) {
        return __ldg(&r[1 + 3 * W]) + __ldg(&r[1 + 2 * W + (idx >> 5)]) + __popc(iw & ((1u << (idx & 31)) - 1u));
    }
};

// raygrid_intersect (main.comp:24-43).
__device__ bool grid_intersect(const RenderArgs& A, float3 o, float3 inv, float& te, float& tl) {
    const float gs = A.world_size;
    float t0x = __fmul_rn(__fsub_rn(__fadd_rn(A.low[0], EPS), o.x), inv.x);
    float t0y = __fmul_rn(__fsub_rn(__fadd_rn(A.low[1], EPS), o.y), inv.y);
    float t0z = __fmul_rn(__fsub_rn(__fadd_rn(A.low[2], EPS), o.z), inv.z);
    float t1x = __fmul_rn(__fsub_rn(__fsub_rn(__fadd_rn(A.low[0], gs), EPS), o.x), inv.x);
    float t1y = __fmul_rn(__fsub_rn(__fsub_rn(__fadd_rn(A.low[1], gs), EPS), o.y), inv.y);
    float t1z = __fmul_rn(__fsub_rn(__fsub_rn(__fadd_rn(A.low[2], gs), EPS), o.z), inv.z);
    if (inv.x < 0.0f) { const float t = t0x; t0x = t1x; t1x = t; }
    if (inv.y < 0.0f) { const float t = t0y; t0y = t1y; t1y = t; }
    if (inv.z < 0.0f) { const float t = t0z; t0z = t1z; t1z = t; }
    te = max_sel(t0x, max_sel(t0y, t0z));
    tl = min_sel(t1x, min_sel(t1y, t1z));
    return te <= tl && tl >= 0.0f;
}

// A ray and where it enters and leaves the grid.
struct Ray {
    float3 o, d, inv;
    float enter, leave;
};
__device__ __forceinline__ bool ray_setup(const RenderArgs& A, float3 o, float3 d, Ray& ray) {
    ray.o = o;
    ray.d = d;
    ray.inv = make_float3(__fdiv_rn(1.0f, d.x), __fdiv_rn(1.0f, d.y), __fdiv_rn(1.0f, d.z));
    return grid_intersect(A, o, ray.inv, ray.enter, ray.leave);
}

// dda (main.comp:46-111), kd-restart. Cell coordinates are clamped to
// [0, dim) and the step count is bounded (both also in the oracle).
//
// Bound by issue and by the length of the chain of one step (a twentieth of a
// frame's warps, those along the surface, take most of its time): the
// reference's two nested loops (walk down, restart at the root) are one, so
// that every trip is one step of every live ray (nested, a lane that restarts
// waits for all lanes of its warp to leave the inner loop); restart and descent
// share the code that enters a level; cell numbers are computed in floats, by
// a sum rounded down at 2^23, without conversions; the divisions by the cell
// size are five operations each with its reciprocal (div_by) instead of a
// general division; the leaf and interior words are read together (the child
// number with them as well was slower, 0.55 against 0.52 ms: more lines).
// 2048^3 scene at 1080p 1.20 -> 0.52 ms, 128 frames of 512^2 6.2 -> 3.2 ms.
template <bool CMP>
__device__ bool dda(const RenderArgs& A, const Level* lv, const Ray& ray, uint4* seen, RHit& hit) {
    constexpr float MAGIC = 0x1p23f;
    constexpr uint32_t CYCLE_FROM = 1024;  // a power of two, above what rays that end take (600)
    const float3 o = ray.o, d = ray.d, inv = ray.inv;
    const float sx = inv.x >= 0.0f ? 1.0f : 0.0f, sy = inv.y >= 0.0f ? 1.0f : 0.0f,
                sz = inv.z >= 0.0f ? 1.0f : 0.0f;
    const uint32_t last = A.levels - 1;
    const float g_leave = ray.leave, g_stop = __fsub_rn(g_leave, EPS);
    // No step before the first restart: t_curr < t_max - EPS does not hold.
    float t_max = __fadd_rn(max_sel(ray.enter, 0.0f), EPS), t_curr = t_max;
    uint32_t steps = 0, lvl = 0, node = 0, W = 0;
    float cs = 1.0f, rcs = 1.0f, vmax = 0.0f, fdim = 0.0f, npx = 0.0f, npy = 0.0f, npz = 0.0f;
    const uint32_t* r = nullptr;
    bool entered = false;
    while (true) {
        if (!(t_curr < __fsub_rn(t_max, EPS))) {  // the node is left: restart at the root
            if (!(t_max < g_stop)) break;
            t_curr = __fadd_rn(t_max, EPS);
            t_max = g_leave;
            if (!(t_curr < g_stop)) break;
            lvl = 0;
            node = 0;
            npx = A.low[0];
            npy = A.low[1];
            npz = A.low[2];
            entered = true;
        }
        if (entered) {
            const Level l = lv[lvl];
            r = node_rec(l, node);
            cs = l.cell;
            rcs = l.rcell;
            vmax = l.vmax;
            fdim = l.dim;
            W = l.words;
        }
        // Rays along cell faces can stop advancing, at one t or around a cycle of
        // cells, and the reference walks them until the step bound (65,536 steps
        // in one warp, 11 to 16 ms). t, the end of the node and the node are all
        // that a step depends on, so a state seen before means that the bound is
        // what ends this ray. Looked for as Brent's method does (against the state
        // saved at the last power of two), and only past CYCLE_FROM steps: 0.33 ms for
        // such a frame of the 4096^3 demo shape, like the others.
        if (steps >= CYCLE_FROM) {
            const uint4 now = make_uint4(__float_as_uint(t_curr), __float_as_uint(t_max), lvl, node);
            const uint4 old = *seen;
            if ((steps & (steps - 1)) == 0) *seen = now;
            else if (now.x == old.x && now.y == old.y && now.z == old.z && now.w == old.w) steps = MAX_DDA_STEPS;
        }
        if (++steps > MAX_DDA_STEPS) break;
        const float te = __fadd_rn(t_curr, EPS);
        const float vx = __fsub_rn(__fadd_rn(o.x, __fmul_rn(te, d.x)), npx);
        const float vy = __fsub_rn(__fadd_rn(o.y, __fmul_rn(te, d.y)), npy);
        const float vz = __fsub_rn(__fadd_rn(o.z, __fmul_rn(te, d.z)), npz);
        float nx = div_by(vx, cs, rcs), ny = div_by(vy, cs, rcs), nz = div_by(vz, cs, rcs);
        if (!(fminf(fminf(fabsf(vx), fabsf(vy)), fabsf(vz)) >= DIV_BY_MIN &&
              fmaxf(fmaxf(fabsf(vx), fabsf(vy)), fabsf(vz)) <= vmax)) {
            // Outside the range, but for zeros, whose sign alone may differ:
            // it reaches no result below.
            const auto fits = [&](float v) { return v == 0.0f ? vmax > 0.0f : fabsf(v) >= DIV_BY_MIN && fabsf(v) <= vmax; };
            if (!(fits(vx) && fits(vy) && fits(vz))) {
                nx = __fdiv_rn(vx, cs);
                ny = __fdiv_rn(vy, cs);
                nz = __fdiv_rn(vz, cs);
            }
        }
        // floor and clamp to [0, dim): clamped first (a NaN gives 0), then
        // MAGIC + v rounded down is MAGIC + floor(v).
        const float top = __fsub_rn(fdim, 1.0f);
        const float cx = __fsub_rn(__fadd_rd(fminf(fmaxf(nx, 0.0f), top), MAGIC), MAGIC);
        const float cy = __fsub_rn(__fadd_rd(fminf(fmaxf(ny, 0.0f), top), MAGIC), MAGIC);
        const float uz = __fadd_rd(fminf(fmaxf(nz, 0.0f), top), MAGIC), cz = __fsub_rn(uz, MAGIC);
        // z + dim y + dim^2 x < 2^15: exact, in the low bits beside MAGIC.
        const uint32_t idx = __float_as_uint(__fmaf_rn(__fmaf_rn(cx, fdim, cy), fdim, uz)) & 0x7FFFFFu;
        const uint32_t leaf = Layout<CMP>::leaf_word(r, W, idx);
        const uint32_t inner = lvl < last ? Layout<CMP>::interior_word(r, W, idx) : 0u;
        const float tnx = __fadd_rn(te, __fmul_rn(__fmul_rn(__fsub_rn(__fadd_rn(cx, sx), nx), cs), inv.x));
        const float tny = __fadd_rn(te, __fmul_rn(__fmul_rn(__fsub_rn(__fadd_rn(cy, sy), ny), cs), inv.y));
        const float tnz = __fadd_rn(te, __fmul_rn(__fmul_rn(__fsub_rn(__fadd_rn(cz, sz), nz), cs), inv.z));
        const float tn = min_sel(tnx, min_sel(tny, tnz));
        if ((leaf >> (idx & 31)) & 1u) {
            hit.t = t_curr;
            hit.node = node;
            hit.level = lvl;
            hit.cell = idx;
            hit.steps = steps;
            return true;
        }
        entered = (inner >> (idx & 31)) & 1u;
        if (entered) {
            node = Layout<CMP>::child(r, W, idx, inner);
            lvl++;
            npx = __fadd_rn(npx, __fmul_rn(cx, cs));
            npy = __fadd_rn(npy, __fmul_rn(cy, cs));
            npz = __fadd_rn(npz, __fmul_rn(cz, cs));
            t_max = tn;
        } else {
            t_curr = tn;
        }
    }
    hit.steps = steps;
    return false;
}

// The gradient of the operations that the common path leaves out.
__device__ __noinline__ float4 gradient_rare(uint32_t op, float4 a, float4 b) {
    switch (op) {
        case OP_SIN: {
            const float c = frep_cosf(a.w);
            return make_float4(__fmul_rn(c, a.x), __fmul_rn(c, a.y), __fmul_rn(c, a.z), frep_sinf(a.w));
        }
        case OP_COS: {
            const float ms = -frep_sinf(a.w);
            return make_float4(__fmul_rn(ms, a.x), __fmul_rn(ms, a.y), __fmul_rn(ms, a.z), frep_cosf(a.w));
        }
        case OP_DIV: {
            const float dd = __fmul_rn(b.w, b.w);
            return make_float4(__fdiv_rn(__fsub_rn(__fmul_rn(a.x, b.w), __fmul_rn(a.w, b.x)), dd),
                               __fdiv_rn(__fsub_rn(__fmul_rn(a.y, b.w), __fmul_rn(a.w, b.y)), dd),
                               __fdiv_rn(__fsub_rn(__fmul_rn(a.z, b.w), __fmul_rn(a.w, b.z)), dd),
                               __fdiv_rn(a.w, b.w));
        }
        case OP_EXP: {
            const float e = frep_expf(a.w);
            return make_float4(__fmul_rn(e, a.x), __fmul_rn(e, a.y), __fmul_rn(e, a.z), e);
        }
        default: {  // SQRT
            const float sq = __fsqrt_rn(a.w);
            const float dd = __fmul_rn(2.0f, sq);
            return make_float4(__fdiv_rn(a.x, dd), __fdiv_rn(a.y, dd), __fdiv_rn(a.z, dd), sq);
        }
    }
}

__device__ __forceinline__ float flip(float v, uint32_t sign) { return __uint_as_float(__float_as_uint(v) ^ sign); }

// tape_eval_gradient (gradient.comp:4-88) with a per-thread slot array of NS
// entries (local memory; in shared memory the slots cost the walk its L1:
// 0.72 against 0.63 ms for the 2048^3 scene at 1080p). The lanes run the tapes
// of different nodes, so a switch over the operation runs most of its arms on
// each trip, each behind the dispatch: the common operations are computed
// together and selected, and the next word is on its way while one runs.
template <int NS>
__device__ float3 gradient(const uint64_t* tape, uint32_t n, float x, float y, float z, float t) {
    constexpr uint32_t RARE = 1u << OP_SIN | 1u << OP_COS | 1u << OP_DIV | 1u << OP_EXP | 1u << OP_SQRT;
    float4 s[NS];
    s[0] = make_float4(1, 0, 0, x);
    s[1] = make_float4(0, 1, 0, y);
    s[2] = make_float4(0, 0, 1, z);
    s[3] = make_float4(0, 0, 0, t);
    uint64_t next = n ? __ldg(&tape[0]) : 0;
    for (uint32_t i = 0; i < n; i++) {
        const uint64_t w = next;
        if (i + 1 < n) next = __ldg(&tape[i + 1]);
        const uint32_t op = w_op(w);
        const float4 a = s[op == OP_CONST ? 0u : w_a(w)], b = s[is_binary(op) ? w_b(w) : 0u];
        float4 r;
        if ((RARE >> op) & 1u) {
            r = gradient_rare(op, a, b);
        } else {
            // ADD, SUB (a + -b), MUL (the product rule), and for the others
            // one operand, its sign flipped for NEG.
            const uint32_t sub = op == OP_SUB ? 0x80000000u : 0u, neg = op == OP_NEG ? 0x80000000u : 0u;
            const bool second = (op == OP_MIN && !(a.w < b.w)) || (op == OP_MAX && !(a.w > b.w));
            const bool mul = op == OP_MUL;
            r.x = mul ? __fadd_rn(__fmul_rn(a.x, b.w), __fmul_rn(a.w, b.x)) : flip(second ? b.x : a.x, neg);
            r.y = mul ? __fadd_rn(__fmul_rn(a.y, b.w), __fmul_rn(a.w, b.y)) : flip(second ? b.y : a.y, neg);
            r.z = mul ? __fadd_rn(__fmul_rn(a.z, b.w), __fmul_rn(a.w, b.z)) : flip(second ? b.z : a.z, neg);
            r.w = mul ? __fmul_rn(a.w, b.w) : flip(second ? b.w : a.w, neg);
            if (op == OP_ADD || op == OP_SUB) {
                r.x = __fadd_rn(a.x, flip(b.x, sub));
                r.y = __fadd_rn(a.y, flip(b.y, sub));
                r.z = __fadd_rn(a.z, flip(b.z, sub));
                r.w = __fadd_rn(a.w, flip(b.w, sub));
            }
            if (op == OP_CONST) r = make_float4(0, 0, 0, w_const(w));
        }
        s[w_out(w)] = r;
    }
    return make_float3(s[0].x, s[0].y, s[0].z);
}

// The same for one tape that all 32 lanes run (each at its own point): the
// lanes decode 32 words at once into `stage` (a warp's 32 records in shared
// memory), and every branch is the warp's.
template <int NS>
__device__ float3 gradient_shared_tape(const uint64_t* tape, uint32_t n, float x, float y, float z, float t,
                                       uint4* stage) {
    const uint32_t lane = threadIdx.x & 31;
    float4 s[NS];
    s[0] = make_float4(1, 0, 0, x);
    s[1] = make_float4(0, 1, 0, y);
    s[2] = make_float4(0, 0, 1, z);
    s[3] = make_float4(0, 0, 0, t);
    uint64_t next = lane < n ? __ldg(&tape[lane]) : 0;
    for (uint32_t base = 0; base < n; base += 32) {
        const uint64_t w = next;
        if (base + 32 + lane < n) next = __ldg(&tape[base + 32 + lane]);
        const uint32_t op = w_op(w);
        __syncwarp();
        stage[lane] = make_uint4(op == OP_CONST ? (uint32_t)(w >> 32) : w_a(w), is_binary(op) ? w_b(w) : 0u, w_out(w), op);
        __syncwarp();
        const uint32_t m = min(n - base, 32u);
        uint4 rec = stage[0];
        for (uint32_t j = 0; j < m; j++) {
            const uint4 q = rec;
            rec = stage[(j + 1) & 31];
            float4 r;
            if (q.w == OP_CONST) {
                r = make_float4(0, 0, 0, __uint_as_float(q.x));
            } else {
                const float4 a = s[q.x], b = s[q.y];
                if (q.w == OP_MUL)
                    r = make_float4(__fadd_rn(__fmul_rn(a.x, b.w), __fmul_rn(a.w, b.x)),
                                    __fadd_rn(__fmul_rn(a.y, b.w), __fmul_rn(a.w, b.y)),
                                    __fadd_rn(__fmul_rn(a.z, b.w), __fmul_rn(a.w, b.z)), __fmul_rn(a.w, b.w));
                else if (q.w == OP_ADD)
                    r = make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z), __fadd_rn(a.w, b.w));
                else if (q.w == OP_SUB)
                    r = make_float4(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z), __fsub_rn(a.w, b.w));
                else if (is_mm(q.w))
                    r = (q.w == OP_MIN ? a.w < b.w : a.w > b.w) ? a : b;
                else if (q.w == OP_NEG)
                    r = make_float4(-a.x, -a.y, -a.z, -a.w);
                else if (q.w == OP_COPY)
                    r = a;
                else
                    r = gradient_rare(q.w, a, b);
            }
            s[q.z] = r;
        }
    }
    return make_float3(s[0].x, s[0].y, s[0].z);
}

// The normals' gradients of a warp: lanes with `need` set have a tape of n
// words. A tape much longer than the others' (a hit on a full cell of the root
// has the whole shape's) runs first, for its lanes alone: in lockstep a word
// costs about 250 cycles, on its own 140 (a warp by itself), so it is taken out
// when the rest then has at most half its trips; a warp with one tape always.
// (A 25,000-word root tape: 3.3 -> 1.8 ms of one warp. Taking every tape out
// that is the longest: 0.65 against 0.59 ms for the 2048^3 scene.)
template <int NS>
__device__ float3 warp_gradient(bool need, const uint64_t* tape, uint32_t n, float3 p, float t, uint4* stage) {
    float3 g = make_float3(0.0f, 0.0f, 0.0f);
    while (true) {
        const uint32_t longest = __reduce_max_sync(~0u, need ? n : 0u);
        if (longest == 0) break;
        const int lead = __ffs(__ballot_sync(~0u, need && n == longest)) - 1;
        const unsigned long long lt = __shfl_sync(~0u, reinterpret_cast<unsigned long long>(tape), lead);
        const bool mine = need && reinterpret_cast<unsigned long long>(tape) == lt;
        if (__reduce_max_sync(~0u, need && !mine ? n : 0u) > longest / 2) break;
        const float3 v = gradient_shared_tape<NS>(reinterpret_cast<const uint64_t*>(lt), longest, p.x, p.y, p.z, t, stage);
        if (mine) {
            g = v;
            need = false;
        }
    }
    if (need) g = gradient<NS>(tape, n, p.x, p.y, p.z, t);
    return g;
}

__device__ __forceinline__ float dot3(float3 a, float3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ float3 normalize3(float3 v) {
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(dot3(v, v)));
    return make_float3(__fmul_rn(v.x, inv), __fmul_rn(v.y, inv), __fmul_rn(v.z, inv));
}

// rand() of random.comp:10-15, with the library's sine.
__device__ __forceinline__ float rand_step(float& seed, uint32_t gx, uint32_t gy) {
    const float dotv = __fadd_rn(__fmul_rn((float)gx, 12.9898f), __fmul_rn((float)gy, 78.233f));
    const float v = __fmul_rn(frep_sinf(__fmul_rn(__fdiv_rn(seed, 100.0f), dotv)), 43758.5453f);
    seed = __fadd_rn(seed, 1.0f);
    return __fsub_rn(v, floorf(v));
}

__device__ __forceinline__ uint8_t to_unorm8(float c) {
    if (!(c > 0.0f)) return 0;
    if (c >= 1.0f) return 255;
    return (uint8_t)__fadd_rn(__fmul_rn(c, 255.0f), 0.5f);
}

struct HitRecord {  // == frep_hit
    float t;
    float n[3];
    uint32_t level, node, cell, steps;
};

template <int NS, bool CMP>
__device__ __forceinline__ void render_pixel(const RenderArgs& A, uint32_t x, uint32_t y, uint32_t layer) {
    __shared__ uint4 stage[RENDER_THREADS];
    __shared__ Level levels[RENDER_THREADS / 32][MAX_LEVELS];
    Level* const lv = levels[threadIdx.x >> 5];
    // Lanes past the image's edge stay for the warp's joint work.
    const bool inside = x < A.width && y < A.height;

    // Ray generation (main.comp:168-178).
    float ox = 0.0f, oy = 0.0f;
    if (A.jitter) {
        float seed = __fadd_rn(A.jitter_seed, (float)layer);
        const float r0 = rand_step(seed, x, y);
        const float r1 = rand_step(seed, x, y);
        ox = __fmul_rn(2.0f, __fsub_rn(r0, 0.5f));
        oy = __fmul_rn(2.0f, __fsub_rn(r1, 0.5f));
    }
    const float dx = __fsub_rn(__fmul_rn(2.0f, __fdiv_rn(__fadd_rn((float)x, ox), (float)A.width)), 1.0f);
    const float dy = __fsub_rn(__fmul_rn(2.0f, __fdiv_rn(__fadd_rn((float)y, oy), (float)A.height)), 1.0f);
    float3 o, d;
    if (A.projection == 0) {
        o = make_float3(A.pos[0], A.pos[1], A.pos[2]);
        const float ax = __fmul_rn(dx, A.sws_x), ay = __fmul_rn(dy, A.sws_y);
        d = normalize3(make_float3(__fadd_rn(__fadd_rn(A.fwd[0], __fmul_rn(ax, A.right[0])), __fmul_rn(ay, A.up[0])),
                                   __fadd_rn(__fadd_rn(A.fwd[1], __fmul_rn(ax, A.right[1])), __fmul_rn(ay, A.up[1])),
                                   __fadd_rn(__fadd_rn(A.fwd[2], __fmul_rn(ax, A.right[2])), __fmul_rn(ay, A.up[2]))));
    } else {
        const float ax = __fmul_rn(dx, A.half_w), ay = __fmul_rn(dy, A.half_h);
        o = make_float3(__fadd_rn(__fadd_rn(A.pos[0], __fmul_rn(ax, A.right[0])), __fmul_rn(ay, A.up[0])),
                        __fadd_rn(__fadd_rn(A.pos[1], __fmul_rn(ax, A.right[1])), __fmul_rn(ay, A.up[1])),
                        __fadd_rn(__fadd_rn(A.pos[2], __fmul_rn(ax, A.right[2])), __fmul_rn(ay, A.up[2])));
        d = make_float3(A.fwd[0], A.fwd[1], A.fwd[2]);
    }

    RHit h;
    h.t = 0.0f;
    h.steps = 0;
    Ray ray;
    bool did = inside && ray_setup(A, o, d, ray);
    if (__ballot_sync(~0u, did)) {
        load_levels<CMP>(A, lv);
        did = did && dda<CMP>(A, lv, ray, stage + threadIdx.x, h);
    }
    const bool lit = did && !(h.t < 0.0f);
    const float px = __fadd_rn(o.x, __fmul_rn(h.t, d.x));
    const float py = __fadd_rn(o.y, __fmul_rn(h.t, d.y));
    const float pz = __fadd_rn(o.z, __fmul_rn(h.t, d.z));
    float3 grad = make_float3(0.0f, 0.0f, 0.0f);
    if (__ballot_sync(~0u, lit)) {
        const uint64_t* tape = nullptr;
        uint32_t tn = 0;
        if (lit) {
            const uint32_t tidx = __ldg(&node_rec(lv[h.level], h.node)[0]);
            tn = (uint32_t)__ldg(&A.tapes[tidx]);
            tape = A.tapes + tidx + 1;
        }
        grad = warp_gradient<NS>(lit, tape, tn, make_float3(px, py, pz), A.tape_time, stage + (threadIdx.x & ~31u));
    }
    if (!inside) return;
    float col[4];
    float3 n = make_float3(0.0f, 0.0f, 0.0f);
    if (!did) {
        for (int c = 0; c < 4; c++) col[c] = A.background[c];
    } else if (h.t < 0.0f) {  // main.comp:149-151
        for (int c = 0; c < 4; c++) col[c] = 1.0f;
    } else {  // shade (main.comp:115-139)
        n = normalize3(grad);
        float diff[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (uint32_t i = 0; i < A.n_lights; i++) {
            const float3 L = make_float3(A.light_dir[i][0], A.light_dir[i][1], A.light_dir[i][2]);
            if (A.shadow_mask & (1u << i)) {
                const float ts = __fsub_rn(h.t, EPS);
                const float3 so = make_float3(__fadd_rn(o.x, __fmul_rn(ts, d.x)), __fadd_rn(o.y, __fmul_rn(ts, d.y)),
                                              __fadd_rn(o.z, __fmul_rn(ts, d.z)));
                RHit sh;
                Ray sr;
                if (ray_setup(A, so, make_float3(-L.x, -L.y, -L.z), sr) && dda<CMP>(A, lv, sr, stage + threadIdx.x, sh)) continue;
            }
            const float dd = dot3(make_float3(-L.x, -L.y, -L.z), n);
            const float inten = fmaxf(dd, 0.0f);
            for (int c = 0; c < 4; c++) diff[c] = __fadd_rn(diff[c], __fmul_rn(inten, A.light_color[i][c]));
        }
        for (int c = 0; c < 4; c++) col[c] = __fadd_rn(A.ambient[c], diff[c]);
    }
    const size_t pix = ((size_t)layer * A.height + y) * A.width + x;
    if (A.rgba8) {
        uchar4 v = make_uchar4(to_unorm8(col[0]), to_unorm8(col[1]), to_unorm8(col[2]), to_unorm8(col[3]));
        reinterpret_cast<uchar4*>(A.rgba8)[pix] = v;
    }
    if (A.hits) {
        HitRecord r;
        r.t = did ? h.t : 0.0f;
        r.n[0] = n.x;
        r.n[1] = n.y;
        r.n[2] = n.z;
        r.level = did ? h.level : 0xFFFFFFFFu;
        r.node = did ? h.node : 0xFFFFFFFFu;
        r.cell = did ? h.cell : 0xFFFFFFFFu;
        r.steps = h.steps;
        reinterpret_cast<HitRecord*>(A.hits)[pix] = r;
    }
}

// blockIdx.z: the layer of a multi-sample image (jitter seeds one apart), whose
// layers follow one another in the outputs.
template <int NS, bool CMP = false>
__global__ void __launch_bounds__(RENDER_THREADS) render_kernel(const RenderArgs A, uint32_t layer0) {
    const uint32_t x = blockIdx.x * 8 + (threadIdx.x & 7);
    const uint32_t y = blockIdx.y * 8 + (threadIdx.x >> 3);
    render_pixel<NS, CMP>(A, x, y, layer0 + blockIdx.z);
}

// Many frames in one launch: blockIdx.z selects the frame.
template <int NS>
__global__ void __launch_bounds__(RENDER_THREADS) render_batch_kernel(const RenderArgs* args) {
    const RenderArgs& A = args[blockIdx.z];
    const uint32_t x = blockIdx.x * 8 + (threadIdx.x & 7);
    const uint32_t y = blockIdx.y * 8 + (threadIdx.x >> 3);
    render_pixel<NS, false>(A, x, y, 0);
}

// Temporal resolve (renderer/triangle.frag:14-23): the pixel is the mean of
// the layers' rgb with alpha 1. The mean is exact (integer sum) and rounded
// to nearest, ties up: (2 sum + n) / 2n; the reference leaves the float ->
// unorm rounding to the driver. One thread per pixel, 4 bytes each.
__global__ void resolve_layers_kernel(const uchar4* __restrict__ layers, uint32_t n, uint32_t pixels,
                                      uchar4* __restrict__ out) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < pixels; p += gridDim.x * blockDim.x) {
        uint32_t r = 0, g = 0, b = 0;
        for (uint32_t i = 0; i < n; i++) {
            const uchar4 v = layers[(size_t)i * pixels + p];
            r += v.x;
            g += v.y;
            b += v.z;
        }
        const uint32_t den = 2 * n;
        out[p] = make_uchar4((uint8_t)((2 * r + n) / den), (uint8_t)((2 * g + n) / den), (uint8_t)((2 * b + n) / den),
                             255);
    }
}

}  // namespace dev

cudaError_t launch_resolve_layers(const uint8_t* layers, uint32_t n, uint32_t pixels, uint8_t* out,
                                  cudaStream_t stream) {
    if (n == 0 || pixels == 0) return cudaSuccess;
    const uint32_t blocks = (uint32_t)std::min<uint64_t>((pixels + 255) / 256, 148ull * 16);
    dev::resolve_layers_kernel<<<blocks, 256, 0, stream>>>(reinterpret_cast<const uchar4*>(layers), n, pixels,
                                                            reinterpret_cast<uchar4*>(out));
    return cudaGetLastError();
}

template <bool CMP>
static void render_launch(const RenderArgs& a, dim3 grid, uint32_t layer0, cudaStream_t stream) {
    constexpr uint32_t T = dev::RENDER_THREADS;
    const uint32_t ns = a.n_slots;
    if (ns <= 32) dev::render_kernel<32, CMP><<<grid, T, 0, stream>>>(a, layer0);
    else if (ns <= 64) dev::render_kernel<64, CMP><<<grid, T, 0, stream>>>(a, layer0);
    else if (ns <= 128) dev::render_kernel<128, CMP><<<grid, T, 0, stream>>>(a, layer0);
    else if (ns <= 256) dev::render_kernel<256, CMP><<<grid, T, 0, stream>>>(a, layer0);
    else if (ns <= 512) dev::render_kernel<512, CMP><<<grid, T, 0, stream>>>(a, layer0);
    else dev::render_kernel<1024, CMP><<<grid, T, 0, stream>>>(a, layer0);
}

cudaError_t launch_render(const RenderArgs& a, cudaStream_t stream, uint32_t layers) {
    if (a.n_slots > 1024) return cudaErrorInvalidValue;
    for (uint32_t at = 0; at < layers; at += 65535) {  // the largest gridDim.z
        const dim3 grid((a.width + 7) / 8, (a.height + 7) / 8, std::min(layers - at, 65535u));
        if (a.compact) render_launch<true>(a, grid, at, stream);
        else render_launch<false>(a, grid, at, stream);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_render_batch(const RenderArgs* args, uint32_t n, uint32_t max_w, uint32_t max_h,
                                uint32_t max_slots, cudaStream_t stream) {
    if (n == 0) return cudaSuccess;
    if (n > 65535 || max_slots > 1024) return cudaErrorInvalidValue;
    constexpr uint32_t T = dev::RENDER_THREADS;
    const dim3 grid((max_w + 7) / 8, (max_h + 7) / 8, n);
    const uint32_t ns = max_slots;
    if (ns <= 32) dev::render_batch_kernel<32><<<grid, T, 0, stream>>>(args);
    else if (ns <= 64) dev::render_batch_kernel<64><<<grid, T, 0, stream>>>(args);
    else if (ns <= 128) dev::render_batch_kernel<128><<<grid, T, 0, stream>>>(args);
    else if (ns <= 256) dev::render_batch_kernel<256><<<grid, T, 0, stream>>>(args);
    else if (ns <= 512) dev::render_batch_kernel<512><<<grid, T, 0, stream>>>(args);
    else dev::render_batch_kernel<1024><<<grid, T, 0, stream>>>(args);
    return cudaGetLastError();
}

}  // namespace frep
