// Tape evaluation on the device over caller-given points and boxes.
//
// frep_tape_eval_device replaces csg::Tape::Eval (vulkan/src/csg/tape.cpp:
// 274-302) for many points at once; frep_tape_eval_intervals exposes the
// interval extension the level passes compute (tape_eval_interval,
// vulkan/shaders/tape/interval.comp:8-160) for arbitrary boxes. Both run the
// same per-instruction device functions as the voxelizer (pt_apply, iv_apply
// in device_common.cuh), so a value or interval returned here is the one a
// level pass computes for the same tape and box. They are what the soundness
// checks of the outward mode measure: every interval must contain the tape's
// value at any point of its box.
//
// One thread per box; the slot file lives in global memory as rows [slot][item]
// (coalesced), allocated per call. Points keep their slots in shared memory
// where a tape's slots fit (eval_points_shared_kernel).
#include <algorithm>
#include <vector>

#include "capi_internal.h"

namespace frep {
namespace dev {

__global__ void eval_points_kernel(const uint64_t* __restrict__ tape, uint32_t n_instr, uint32_t n_slots,
                                   const float4* __restrict__ xyzt, uint32_t n, float* __restrict__ slots,
                                   float* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = xyzt[i];
    // point.comp:4-7: slots 0..3 = x, y, z, t
    slots[0 * (size_t)n + i] = p.x;
    slots[1 * (size_t)n + i] = p.y;
    slots[2 * (size_t)n + i] = p.z;
    slots[3 * (size_t)n + i] = p.w;
    for (uint32_t j = 0; j < n_instr; j++) {
        const uint64_t w = __ldg(&tape[j]);
        const uint32_t op = w_op(w);
        const float a = op == OP_CONST ? 0.0f : slots[(size_t)w_a(w) * n + i];
        const float b = is_binary(op) ? slots[(size_t)w_b(w) * n + i] : 0.0f;
        slots[(size_t)w_out(w) * n + i] = pt_apply(op, w, a, b);
    }
    out[i] = slots[i];
    (void)n_slots;
}

// Points with the slot file in shared memory, K per thread (rows of K floats,
// [row][thread]: one access of up to 16 bytes per operand), over records that
// the host makes of the tape (point_code: constants in the words that use them,
// few rows), every branch the warp's. In global memory each word costs three accesses of the whole file
// (270 MB for a million points and the 67 slots of a union of 64 spheres), and
// the file has to be allocated: 1.61 -> 0.30 ms (with 13 slots and 2,900 words
// 5.2 -> 0.90 ms), a thousand points 158 -> 48 us.
constexpr uint32_t EVAL_THREADS = 64, EVAL_MAX_ROWS = 48;
// A record: operand a, operand b (offset of the row, or a constant's bits), the
// result's row, the operation with these bits.
constexpr uint32_t EVAL_IMM_A = 1u << 8, EVAL_IMM_B = 1u << 9;

template <int K>
struct alignas(4 * K) Points {
    float v[K];
};

// The operations that the loop below leaves out.
template <int K>
__device__ __noinline__ Points<K> eval_rare(uint32_t op, Points<K> a, Points<K> b) {
#pragma unroll 1
    for (int k = 0; k < K; k++) a.v[k] = pt_apply(op, 0, a.v[k], b.v[k]);
    return a;
}

template <int K>
__global__ void __launch_bounds__(EVAL_THREADS)
    eval_points_shared_kernel(const uint4* __restrict__ recs, uint32_t n_recs, uint32_t result,
                              const float4* __restrict__ xyzt, uint32_t n, float* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char eval_shared[];
    uint4* const stage = reinterpret_cast<uint4*>(eval_shared) + (threadIdx.x & ~31u);
    Points<K>* const s = reinterpret_cast<Points<K>*>(eval_shared + EVAL_THREADS * sizeof(uint4)) + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t first = (uint64_t)blockIdx.x * (EVAL_THREADS * K) + threadIdx.x;
#pragma unroll
    for (int k = 0; k < K; k++) {
        const uint64_t i = first + (uint64_t)k * EVAL_THREADS;
        const float4 p = xyzt[i < n ? i : n - 1];
        s[0 * EVAL_THREADS].v[k] = p.x;
        s[1 * EVAL_THREADS].v[k] = p.y;
        s[2 * EVAL_THREADS].v[k] = p.z;
        s[3 * EVAL_THREADS].v[k] = p.w;
    }
    uint4 next = lane < n_recs ? __ldg(&recs[lane]) : make_uint4(0, 0, 0, 0);
    for (uint32_t base = 0; base < n_recs; base += 32) {
        __syncwarp();
        stage[lane] = next;
        __syncwarp();
        if (base + 32 + lane < n_recs) next = __ldg(&recs[base + 32 + lane]);
        const uint32_t m = min(n_recs - base, 32u);
        uint4 rec = stage[0];
        for (uint32_t j = 0; j < m; j++) {
            const uint4 q = rec;
            rec = stage[(j + 1) & 31];
            const uint32_t op = q.w & 0xFFu;
            Points<K> a = s[q.w & EVAL_IMM_A ? 0u : q.x], b = s[q.w & EVAL_IMM_B ? 0u : q.y];
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (q.w & EVAL_IMM_A) a.v[k] = __uint_as_float(q.x);
                if (q.w & EVAL_IMM_B) b.v[k] = __uint_as_float(q.y);
            }
            Points<K> r;
            if (op == OP_MUL) {
#pragma unroll
                for (int k = 0; k < K; k++) r.v[k] = pt_apply(OP_MUL, 0, a.v[k], b.v[k]);
            } else if (op == OP_ADD) {
#pragma unroll
                for (int k = 0; k < K; k++) r.v[k] = pt_apply(OP_ADD, 0, a.v[k], b.v[k]);
            } else if (op == OP_SUB) {
#pragma unroll
                for (int k = 0; k < K; k++) r.v[k] = pt_apply(OP_SUB, 0, a.v[k], b.v[k]);
            } else if (op == OP_MIN) {
#pragma unroll
                for (int k = 0; k < K; k++) r.v[k] = pt_apply(OP_MIN, 0, a.v[k], b.v[k]);
            } else if (op == OP_MAX) {
#pragma unroll
                for (int k = 0; k < K; k++) r.v[k] = pt_apply(OP_MAX, 0, a.v[k], b.v[k]);
            } else if (op == OP_NEG) {
#pragma unroll
                for (int k = 0; k < K; k++) r.v[k] = pt_apply(OP_NEG, 0, a.v[k], b.v[k]);
            } else {
                r = eval_rare<K>(op, a, b);
            }
            s[q.z] = r;
        }
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
        const uint64_t i = first + (uint64_t)k * EVAL_THREADS;
        if (i < n) out[i] = s[result].v[k];
    }
}

template <int ROUND>
__global__ void eval_intervals_kernel(const uint64_t* __restrict__ tape, uint32_t n_instr,
                                      const float* __restrict__ boxes, uint32_t n, float tape_time,
                                      float2* __restrict__ slots, float2* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* b6 = boxes + 6 * (size_t)i;
    // interval.comp:121-128: slots 0..3 = X, Y, Z over the box, T = [t, t]
    slots[0 * (size_t)n + i] = make_float2(b6[0], b6[3]);
    slots[1 * (size_t)n + i] = make_float2(b6[1], b6[4]);
    slots[2 * (size_t)n + i] = make_float2(b6[2], b6[5]);
    slots[3 * (size_t)n + i] = make_float2(tape_time, tape_time);
    for (uint32_t j = 0; j < n_instr; j++) {
        const uint64_t w = __ldg(&tape[j]);
        const uint32_t op = w_op(w);
        const float2 a = op == OP_CONST ? make_float2(0.0f, 0.0f) : slots[(size_t)w_a(w) * n + i];
        const float2 b = is_binary(op) ? slots[(size_t)w_b(w) * n + i] : make_float2(0.0f, 0.0f);
        slots[(size_t)w_out(w) * n + i] = iv_apply<ROUND>(op, w, a, b);
    }
    out[i] = slots[i];
}

// The hybrid affine mode (FREP_ROUND_HYBRID): each slot row holds the
// interval and the affine form, 8 floats (lo, hi, c, x | y, z, e, 0).
__global__ void eval_hybrid_kernel(const uint64_t* __restrict__ tape, uint32_t n_instr,
                                   const float* __restrict__ boxes, uint32_t n, float tape_time,
                                   float4* __restrict__ slots, float2* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* b6 = boxes + 6 * (size_t)i;
    auto row = [&](uint32_t s) { return slots + 2 * ((size_t)s * n + i); };
    for (int k = 0; k < 3; k++) {
        const Af f = af_axis(b6[k], b6[3 + k], k);
        row(k)[0] = make_float4(b6[k], b6[3 + k], f.c, f.x);
        row(k)[1] = make_float4(f.y, f.z, f.e, 0.0f);
    }
    row(3)[0] = make_float4(tape_time, tape_time, tape_time, 0.0f);
    row(3)[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (uint32_t j = 0; j < n_instr; j++) {
        const uint64_t w = __ldg(&tape[j]);
        const uint32_t op = w_op(w);
        float2 v;
        Af f;
        if (op == OP_CONST) {
            v = make_float2(w_const(w), w_const(w));
            f = Af{v.x, 0.0f, 0.0f, 0.0f, 0.0f};
        } else {
            const uint32_t sb = is_binary(op) ? w_b(w) : 0u;
            const float4 a0 = row(w_a(w))[0], a1 = row(w_a(w))[1];
            const float4 b0 = row(sb)[0], b1 = row(sb)[1];
            const float2 a = make_float2(a0.x, a0.y), b = make_float2(b0.x, b0.y);
            const Af fa{a0.z, a0.w, a1.x, a1.y, a1.z}, fb{b0.z, b0.w, b1.x, b1.y, b1.z};
            const uint32_t c = is_mm(op) ? mm_choice(op, a, b) : 0u;
            v = hy_apply(op, w, a, b, fa, fb, op == OP_MUL && w_a(w) == w_b(w), c, &f);
        }
        row(w_out(w))[0] = make_float4(v.x, v.y, f.c, f.x);
        row(w_out(w))[1] = make_float4(f.y, f.z, f.e, 0.0f);
    }
    out[i] = make_float2(row(0)[0].x, row(0)[0].y);
}

}  // namespace dev
}  // namespace frep

using frep::detail::align_up;
using frep::detail::cuda_fail;
using frep::detail::fail;

namespace {

// Device buffers of one evaluation call, released on every path.
struct EvalBuffers {
    void* p = nullptr;
    ~EvalBuffers() {
        if (p) cudaFree(p);
    }
};

// Every slot an instruction names must be a row of the slot file the kernels
// index with it.
frep_status check_slots(const frep_tape* tape, const char* who) {
    const uint32_t n_slots = std::max<uint32_t>(tape->ct.n_slots, 4);
    for (const uint64_t w : tape->ct.instrs) {
        const uint32_t op = (uint32_t)w & 0xFFu, o = ((uint32_t)w >> 16) & 0xFFFFu;
        const uint32_t a = (uint32_t)(w >> 32) & 0xFFFFu, b = (uint32_t)(w >> 48);
        if (op > FREP_TAPE_COPY || o >= n_slots || (op != FREP_TAPE_CONST && a >= n_slots) ||
            (frep::dev::is_binary(op) && b >= n_slots))
            return fail(FREP_ERR_INVALID_ARG, "%s: instruction names a slot outside the tape's %u slots", who, n_slots);
    }
    return FREP_OK;
}

// The records of eval_points_shared_kernel for a checked tape: the same
// operations on the same operands, without words for constants, in an order
// that keeps few values at a time (operands right before their use, the one
// that needs more rows first) and with rows given out by last use. A tape puts
// the 64 spheres of a union first and their minima last: 67 slots, 9 rows.
struct PointCode {
    std::vector<uint4> recs;
    uint32_t rows = 4, result = 0;  // rows of the slot file, offset of the result's
};

// Stops, with rows above EVAL_MAX_ROWS, at the record that would need as many.
PointCode point_code(const std::vector<uint64_t>& instrs, uint32_t n_slots) {
    constexpr uint32_t T = frep::dev::EVAL_THREADS, CONST = ~0u, INPUTS = 4;
    struct Ref {
        uint32_t value = CONST, bits = 0;  // a value's number, or a constant
    };
    struct Value {
        uint32_t op = 0, need = 0, uses = 0, row = 0;
        Ref a, b;
        bool placed = false;
    };
    std::vector<Value> v;
    v.reserve(INPUTS + instrs.size() + 1);
    v.resize(INPUTS);
    std::vector<Ref> slot(n_slots);
    for (uint32_t i = 0; i < INPUTS; i++) {
        slot[i].value = i;
        v[i].row = i;
        v[i].placed = true;
    }
    for (const uint64_t w : instrs) {
        const uint32_t op = (uint32_t)w & 0xFFu, o = ((uint32_t)w >> 16) & 0xFFFFu;
        if (op == FREP_TAPE_CONST) {
            slot[o] = Ref{CONST, (uint32_t)(w >> 32)};
            continue;
        }
        Value x;
        x.op = op;
        x.a = slot[(uint32_t)(w >> 32) & 0xFFFFu];
        if (frep::dev::is_binary(op)) x.b = slot[(uint32_t)(w >> 48)];
        const uint32_t na = x.a.value == CONST ? 0 : v[x.a.value].need, nb = x.b.value == CONST ? 0 : v[x.b.value].need;
        x.need = std::max(1u, na == nb ? na + 1 : std::max(na, nb));
        slot[o] = Ref{(uint32_t)v.size(), 0};
        v.push_back(x);
    }
    if (slot[0].value < INPUTS || slot[0].value == CONST) {  // no operation left: copy it
        Value x;
        x.op = FREP_TAPE_COPY;
        x.a = slot[0];
        slot[0] = Ref{(uint32_t)v.size(), 0};
        v.push_back(x);
    }
    // How often the result's values are used (operands come before their user).
    const uint32_t result = slot[0].value;
    for (uint32_t i = result; i >= INPUTS; i--) {
        if (i != result && v[i].uses == 0) continue;
        for (const uint32_t u : {v[i].a.value, v[i].b.value})
            if (u != CONST) v[u].uses++;
    }
    // Depth first from the result.
    PointCode code;
    code.recs.reserve(v.size());
    std::vector<uint32_t> stack = {result}, free_rows;
    while (!stack.empty()) {
        const uint32_t i = stack.back();
        Value& x = v[i];
        if (x.placed) {
            stack.pop_back();
            continue;
        }
        const uint32_t a = x.a.value, b = x.b.value;
        const bool wait_a = a != CONST && !v[a].placed, wait_b = b != CONST && !v[b].placed;
        if (wait_a || wait_b) {  // the top of the stack is placed first
            const bool a_first = wait_a && (!wait_b || v[a].need >= v[b].need);
            if (a_first && wait_b) stack.push_back(b);
            if (wait_a) stack.push_back(a);
            if (!a_first && wait_b) stack.push_back(b);
            continue;
        }
        stack.pop_back();
        x.placed = true;
        uint4 q = make_uint4(x.a.bits, x.b.bits, 0, x.op);
        if (a == CONST) q.w |= frep::dev::EVAL_IMM_A;
        else q.x = v[a].row * T;
        if (!frep::dev::is_binary(x.op)) q.y = 0;
        else if (b == CONST) q.w |= frep::dev::EVAL_IMM_B;
        else q.y = v[b].row * T;
        for (const uint32_t u : {a, b})
            if (u != CONST && --v[u].uses == 0 && u >= INPUTS) free_rows.push_back(v[u].row);
        if (free_rows.empty()) {
            x.row = code.rows++;
            if (code.rows > frep::dev::EVAL_MAX_ROWS) return code;
        } else {
            x.row = free_rows.back();
            free_rows.pop_back();
        }
        q.z = x.row * T;
        code.recs.push_back(q);
    }
    code.result = v[result].row * T;
    return code;
}

// `code`: what the kernel runs (the tape's words, or records made of them).
frep_status eval_common(frep_ctx* ctx, const void* code, uint64_t code_bytes, uint64_t in_bytes, uint64_t slot_bytes,
                        uint64_t out_bytes, EvalBuffers* buf, uint8_t** in, uint8_t** slots, uint8_t** out,
                        const char* who) {
    const uint64_t tape_bytes = align_up(code_bytes + 8, 256);
    const uint64_t total = tape_bytes + align_up(in_bytes, 256) + align_up(slot_bytes, 256) + align_up(out_bytes, 256);
    if (!frep::detail::reserve(ctx, total))
        return fail(FREP_ERR_OOM, "%s: %llu bytes of working memory exceed the context's budget", who,
                    (unsigned long long)total);
    FREP_CUDA(cudaSetDevice(ctx->device));
    cudaError_t e = frep::detail::device_alloc(ctx, &buf->p, total);
    if (e != cudaSuccess) {
        buf->p = nullptr;
        return fail(FREP_ERR_OOM, "%s: cudaMalloc of %llu bytes failed (%s)", who, (unsigned long long)total,
                    cudaGetErrorString(e));
    }
    uint8_t* base = static_cast<uint8_t*>(buf->p);
    FREP_CUDA(cudaMemcpy(base, code, code_bytes, cudaMemcpyHostToDevice));
    *in = base + tape_bytes;
    *slots = *in + align_up(in_bytes, 256);
    *out = *slots + align_up(slot_bytes, 256);
    return FREP_OK;
}

}  // namespace

extern "C" frep_status frep_tape_eval_device(frep_ctx* ctx, const frep_tape* tape, const float* xyzt, uint32_t n,
                                             float* out) {
    if (!ctx || !tape || (n && (!xyzt || !out))) return fail(FREP_ERR_INVALID_ARG, "frep_tape_eval_device: null argument");
    if (n == 0) return FREP_OK;
    if (tape->ct.instrs.empty()) return fail(FREP_ERR_INVALID_ARG, "frep_tape_eval_device: empty tape");
    const uint32_t n_slots = std::max<uint32_t>(tape->ct.n_slots, 4);
    // Rows in shared memory while four blocks of four points per thread fit an
    // SM (48 rows: 49 KB each); one point per thread until that many points
    // give each SM two blocks of four (1,000 points: 48 against 66 us with four;
    // 75,776: 68 and 67; 150,000: 110 against 76).
    constexpr uint32_t T = frep::dev::EVAL_THREADS;
    frep_status st = check_slots(tape, "frep_tape_eval_device");
    if (st != FREP_OK) return st;
    const PointCode pc = point_code(tape->ct.instrs, n_slots);
    const bool shared = pc.rows <= frep::dev::EVAL_MAX_ROWS;
    const uint32_t K = n >= (uint64_t)ctx->sm_count * 2 * T * 4 ? 4 : 1;
    EvalBuffers buf;
    uint8_t *d_in, *d_slots, *d_out;
    const void* code = shared ? static_cast<const void*>(pc.recs.data()) : tape->ct.instrs.data();
    const uint64_t code_bytes = shared ? pc.recs.size() * sizeof(uint4) : tape->ct.instrs.size() * 8;
    st = eval_common(ctx, code, code_bytes, (uint64_t)n * 16, shared ? 0 : (uint64_t)n * n_slots * 4, (uint64_t)n * 4,
                     &buf, &d_in, &d_slots, &d_out, "frep_tape_eval_device");
    if (st != FREP_OK) return st;
    FREP_CUDA(cudaMemcpy(d_in, xyzt, (size_t)n * 16, cudaMemcpyHostToDevice));
    const auto* d_xyzt = reinterpret_cast<const float4*>(d_in);
    if (shared) {
        const uint32_t blocks = (uint32_t)(((uint64_t)n + T * K - 1) / (T * K));
        const uint32_t bytes = T * 16 + pc.rows * T * K * 4;
        const auto kernel = K == 4 ? frep::dev::eval_points_shared_kernel<4> : frep::dev::eval_points_shared_kernel<1>;
        FREP_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(T * 16 + frep::dev::EVAL_MAX_ROWS * T * K * 4)));
        kernel<<<blocks, T, bytes>>>(static_cast<const uint4*>(buf.p), (uint32_t)pc.recs.size(), pc.result, d_xyzt,
                                     n, reinterpret_cast<float*>(d_out));
    } else {
        const uint32_t threads = 128, blocks = (n + threads - 1) / threads;
        frep::dev::eval_points_kernel<<<blocks, threads>>>(static_cast<const uint64_t*>(buf.p),
                                                            (uint32_t)tape->ct.instrs.size(), n_slots, d_xyzt, n,
                                                            reinterpret_cast<float*>(d_slots),
                                                            reinterpret_cast<float*>(d_out));
    }
    FREP_CUDA(cudaGetLastError());
    FREP_CUDA(cudaMemcpy(out, d_out, (size_t)n * 4, cudaMemcpyDeviceToHost));
    return FREP_OK;
}

extern "C" frep_status frep_tape_eval_intervals(frep_ctx* ctx, const frep_tape* tape, const float* boxes, uint32_t n,
                                                float tape_time, uint32_t rounding, float* out) {
    if (!ctx || !tape || (n && (!boxes || !out)))
        return fail(FREP_ERR_INVALID_ARG, "frep_tape_eval_intervals: null argument");
    if (rounding > FREP_ROUND_HYBRID) return fail(FREP_ERR_INVALID_ARG, "frep_tape_eval_intervals: rounding %u", rounding);
    if (n == 0) return FREP_OK;
    if (tape->ct.instrs.empty()) return fail(FREP_ERR_INVALID_ARG, "frep_tape_eval_intervals: empty tape");
    const uint32_t n_slots = std::max<uint32_t>(tape->ct.n_slots, 4);
    EvalBuffers buf;
    uint8_t *d_in, *d_slots, *d_out;
    const uint64_t row_bytes = rounding == FREP_ROUND_HYBRID ? 32 : 8;
    frep_status st = check_slots(tape, "frep_tape_eval_intervals");
    if (st != FREP_OK) return st;
    st = eval_common(ctx, tape->ct.instrs.data(), tape->ct.instrs.size() * 8, (uint64_t)n * 24,
                     (uint64_t)n * n_slots * row_bytes, (uint64_t)n * 8, &buf, &d_in, &d_slots, &d_out,
                     "frep_tape_eval_intervals");
    if (st != FREP_OK) return st;
    FREP_CUDA(cudaMemcpy(d_in, boxes, (size_t)n * 24, cudaMemcpyHostToDevice));
    const uint32_t threads = 128, blocks = (n + threads - 1) / threads;
    const auto* t = static_cast<const uint64_t*>(buf.p);
    const uint32_t ni = (uint32_t)tape->ct.instrs.size();
    if (rounding == FREP_ROUND_HYBRID)
        frep::dev::eval_hybrid_kernel<<<blocks, threads>>>(t, ni, reinterpret_cast<const float*>(d_in), n, tape_time,
                                                           reinterpret_cast<float4*>(d_slots),
                                                           reinterpret_cast<float2*>(d_out));
    else if (rounding == FREP_ROUND_OUTWARD)
        frep::dev::eval_intervals_kernel<1><<<blocks, threads>>>(t, ni, reinterpret_cast<const float*>(d_in), n,
                                                                  tape_time, reinterpret_cast<float2*>(d_slots),
                                                                  reinterpret_cast<float2*>(d_out));
    else
        frep::dev::eval_intervals_kernel<0><<<blocks, threads>>>(t, ni, reinterpret_cast<const float*>(d_in), n,
                                                                  tape_time, reinterpret_cast<float2*>(d_slots),
                                                                  reinterpret_cast<float2*>(d_out));
    FREP_CUDA(cudaGetLastError());
    FREP_CUDA(cudaMemcpy(out, d_out, (size_t)n * 8, cudaMemcpyDeviceToHost));
    return FREP_OK;
}
