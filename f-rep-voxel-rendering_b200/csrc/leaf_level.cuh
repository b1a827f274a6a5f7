// The last-level pass over micro-ops (leaf_level_kernel); included by
// voxelizer.cu inside namespace frep::dev, after the point pass, whose results
// it shares bit for bit (FK, lds_k, sts_k, pt_exec's arithmetic).
//
// What bounds the pass is the interpreter: the point pass spent 21 warp
// instructions and 5.7 shared-memory wavefronts per tape instruction on 64
// cells, at 62 % of the issue slots and 67 % of the shared-memory bandwidth.
// Here
//   * the tape runs as micro-ops (micro_ops.h), a third of its words;
//   * leaves with the same tape share its decoding and run it together, 128
//     cells at a time: a warp takes up to 128 consecutive dim-4 nodes and groups
//     32 of them at a time by tape (siblings are neighbours in the node order,
//     and most of them share their parent's shortened tape);
//   * up to 32 tapes are decoded at once, one per lane, each lane going through
//     its tape word by word (75 instructions for a word of 32 tapes), which
//     computes constants on the way; a few tapes are decoded one after the other
//     with their words spread over the lanes, which only folds the next word's;
//   * slot rows are numbered over the slots that the micro-ops read or write as
//     rows, so a tape that names 28 slots but keeps 8 of them in rows takes 8.
// The code that a warp goes through stays small: with an 8-cell loop beside
// these two, unrolled decoders or the rare opcodes in line, a fifth to a half of
// the instruction fetches missed the SM's instruction cache and the pass took
// up to ten times as long.

// A warp's shared memory: its slot rows (while decoding: the constants in the
// slots of each lane's tape), then the staged micro-ops with the end mark, then
// the jobs (distinct tapes) of the items it took.
constexpr uint32_t LEAF_OPS = 128, LEAF_ITEMS = 128;
// From this many tapes on, each lane decodes one of its own. (With 2 instead of
// 10 the 128-scene batch's level-1 pass over dim-4 leaves took 2.3 ms, not 0.9,
// and the 2048^3 scene's pass 2.8, not 2.3; with 4, 2 % more than with 10.)
constexpr uint32_t LEAF_SERIAL = 10;
constexpr uint32_t LEAF_FIXED_BYTES = (LEAF_OPS + 1) * 16 + LEAF_ITEMS * 4;
constexpr uint32_t LEAF_MAX_SLOTS = micro::MO_SLOTS;
constexpr uint32_t LEAF_MIN_ROWS = LEAF_MAX_SLOTS * 128;  // bytes of the decoder's constants

// Items per node of the pass, 8 mask words each (dim 4: the node's two).
__host__ __device__ inline uint32_t leaf_units(uint32_t dim) { return dim == 4 ? 1u : (dim * dim * dim / 32u + 7u) / 8u; }

// leaf_rule.h for a tree at its last level, in a launch of `cells` cells.
__device__ __forceinline__ bool leaf_pays(const TreeHeader* H, uint32_t L, unsigned long long cells) {
    return frep::leaf_pays(H->dims[L], H->transcendental != 0u, H->tape_size_sum[0],
                           H->tape_size_sum[L] / max(1u, H->node_count[L]), cells);
}

#include "leaf_dispatch.cuh"

// One micro-op that the loop leaves to C++, out of line, two cells at a time:
// its double-precision polynomials unrolled over the cells would take the
// kernel's registers and the instruction cache.
template <int K>
__device__ __noinline__ FK<K> leaf_rare(uint4 d, uint32_t lane_base, FK<K> r) {
    const uint32_t op = micro::mo_x_op(d.w), ka = micro::mo_kind_a(d.w), kb = micro::mo_kind_b(d.w);
    FK<K> a = r, b = r;  // forwarded unless
    if (ka == micro::KIND_S) a = lds_k<K>(lane_base + d.x);
    if (op == micro::M_DIV && kb == micro::KIND_S) b = lds_k<K>(lane_base + d.y);
#pragma unroll
    for (int k = 0; k < K; k++) {
        if (ka == micro::KIND_I) a.v[k] = __uint_as_float(d.x);
        if (kb == micro::KIND_I) b.v[k] = __uint_as_float(d.y);
    }
#pragma unroll 1
    for (int i = 0; i < K; i += 2) {
        float x = a.v[0], y = a.v[1];
        if (op == micro::M_DIV) {
            x = __fdiv_rn(x, b.v[0]);
            y = __fdiv_rn(y, b.v[1]);
        } else if (op == micro::M_SQRT) {
            x = __fsqrt_rn(x);
            y = __fsqrt_rn(y);
        } else if (op == micro::M_EXP) {
            x = frep_expf(x);
            y = frep_expf(y);
        } else {
            const int quarter = op == micro::M_COS ? 1 : 0;
            x = frep_sin_quarter(x, quarter);
            y = frep_sin_quarter(y, quarter);
        }
#pragma unroll
        for (int k = 0; k + 2 < K; k++) {
            a.v[k] = a.v[k + 2];
            b.v[k] = b.v[k + 2];
            r.v[k] = r.v[k + 2];
        }
        r.v[K - 2] = x;
        r.v[K - 1] = y;
    }
    if (!(d.w & micro::MO_NO_STORE)) sts_k<K>(lane_base + d.z, r);
    return r;
}

// Runs the staged micro-ops on K cells per lane: the jump-table loop, and
// DIV / SQRT / SIN / COS / EXP in leaf_rare.
template <int K>
__device__ __forceinline__ void leaf_exec(uint32_t at, uint32_t lane_base, FK<K>& r) {
    while (true) {
        LeafRun<K> run;
        if constexpr (K == 2) run = leaf_run_2(at, lane_base, r);
        else run = leaf_run_4(at, lane_base, r);
        r = run.r;
        const uint4 d = lds_u4(run.at);
        if (micro::mo_x_op(d.w) == micro::M_END) return;
        r = leaf_rare<K>(d, lane_base, r);
        at = run.at + 16;
    }
}

// The tape that a warp runs (all lanes alike): its micro-ops, in the warp's
// scratch (`ops` of them) and, when they are few enough, staged.
struct LeafTape {
    const uint64_t* saved;
    uint32_t ops;
    uint32_t mask;    // slots with a row
    uint32_t stride;  // bytes per row
};

// Stages the micro-ops from `at` on as {y, z, w, x}: operands (row offsets, or
// the constant's bits), the output's row offset, the dispatch index; rows of
// `stride` bytes are numbered over the slots in `mask`. Then the end mark.
// Returns where they end.
__device__ __forceinline__ uint32_t leaf_stage(const LeafTape& tp, uint4* stage, uint32_t at, uint32_t lane) {
    const uint32_t m = min(LEAF_OPS, tp.ops - at);
    auto row = [&](uint32_t s) { return (uint32_t)__popc(tp.mask & ((1u << s) - 1u)) * tp.stride; };
    __syncwarp();
#pragma unroll 1
    for (uint32_t i = lane; i < m; i += 32) {
        const uint64_t u = __ldcg(&tp.saved[at + i]);
        const uint32_t lo = (uint32_t)u, imm = (uint32_t)(u >> 32), x = lo & micro::MO_X;
        const bool ia = micro::mo_kind_a(x) == micro::KIND_I || micro::mo_x_op(x) == micro::M_CONST;
        stage[i] = make_uint4(ia ? imm : row(micro::mo_slot_a(lo)),
                              micro::mo_kind_b(x) == micro::KIND_I ? imm : row(micro::mo_slot_b(lo)),
                              row(micro::mo_slot_out(lo)), x);
    }
    if (lane == 0) stage[m] = make_uint4(0u, 0u, 0u, micro::M_END << 4);
    __syncwarp();
    return at + m;
}

// Decodes one tape with its words spread over the lanes (decode_single), to
// `to`. Returns the number of micro-ops and the slots with rows.
__device__ __noinline__ uint2 leaf_decode_one(const uint64_t* rec, uint32_t n, uint64_t* to, uint32_t lane) {
    uint32_t ops = 0, rows = 0;
    // the words one and two before lane 0's: before the tape, ones that wrote no slot
    uint32_t c1 = 0xFFFF0000u, c1_hi = 0u, c2 = 0xFFFF0000u;
    uint64_t w = lane < n ? __ldcg(&rec[1 + lane]) : 0ull;
#pragma unroll 1
    for (uint32_t base = 0; base < n; base += 32) {
        const uint64_t next = base + 32 + lane < n ? __ldcg(&rec[1 + base + 32 + lane]) : 0ull;
        const uint32_t lo = (uint32_t)w, hi = (uint32_t)(w >> 32);
        uint32_t p1 = __shfl_up_sync(0xFFFFFFFFu, lo, 1), p1_hi = __shfl_up_sync(0xFFFFFFFFu, hi, 1);
        uint32_t p2 = __shfl_up_sync(0xFFFFFFFFu, lo, 2);
        if (lane == 0) {
            p1 = c1;
            p1_hi = c1_hi;
            p2 = c2;
        } else if (lane == 1) {
            p2 = c1;
        }
        c1 = __shfl_sync(0xFFFFFFFFu, lo, 31);
        c1_hi = __shfl_sync(0xFFFFFFFFu, hi, 31);
        c2 = __shfl_sync(0xFFFFFFFFu, lo, 30);
        const bool there = base + lane < n && !(lo & (uint32_t)micro::MARK_FOLD);
        const bool gone = there && lane > 0 && micro::elided(w, p1);
        const uint32_t kb = __ballot_sync(0xFFFFFFFFu, there && !gone), eb = __ballot_sync(0xFFFFFFFFu, gone);
        const uint32_t renamed = __ffs(~(eb >> lane >> 1)) - 1u;  // elided words right after this one
        const uint32_t dest = __shfl_sync(0xFFFFFFFFu, lo, (lane + renamed) & 31u);
        if (there && !gone)
            __stcg(&to[ops + __popc(kb & lanemask_lt())],
                   micro::decode_single(w, p1, p1_hi, ((p1 & (uint32_t)micro::MARK_FOLD) ? p2 : p1) >> 16, dest, &rows));
        ops += __popc(kb);
        w = next;
    }
    return make_uint2(ops, __reduce_or_sync(0xFFFFFFFFu, rows));
}

// Decodes up to 32 tapes, lane l the record at `rec` (null: none), to `to` (room
// for as many micro-ops as the tape has words). values: shared address of the
// lane's column of constants (rows of 128 bytes). Returns the number of
// micro-ops, *rows the slots with rows.
__device__ __noinline__ uint32_t leaf_decode(const uint64_t* rec, uint64_t* to, uint32_t values, uint32_t* rows) {
    micro::Decoder d;
    uint32_t n = 0, ops = 0;
    uint64_t w = 0;
    if (rec) {
        n = (uint32_t)rec[0];
        w = rec[1];
    }
    auto value = [&](uint32_t s) {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(values + s * 128u));
        return v;
    };
    auto keep = [&](uint32_t s, uint32_t v) {
        asm volatile("st.shared.u32 [%0], %1;" ::"r"(values + s * 128u), "r"(v) : "memory");
    };
    auto emit = [&](uint32_t lo, uint32_t imm) { __stcg(&to[ops++], (uint64_t)imm << 32 | lo); };
#pragma unroll 1
    for (uint32_t i = 0; i < n; i++) {
        const uint64_t next = i + 1 < n ? rec[i + 2] : 0ull;  // (one word early, its line 16 words early)
        if ((i & 15u) == 0u && i + 32 < n) asm volatile("prefetch.global.L1 [%0];" ::"l"(rec + i + 32));
        micro::decode_word(d, w, value, keep, emit);
        w = next;
    }
    if (n) micro::decode_end(d, emit);
    *rows = d.rows;
    return ops;
}

// low + n * cell size of two cells along one axis. (Not with the packed f32x2
// operations: mul.rn and add.rn of one block gave other bits than apart.)
__device__ __forceinline__ float2 cell_low(float n, float2 c, float low, float cs) {
    return make_float2(__fadd_rn(low, __fmul_rn(__fadd_rn(n, c.x), cs)),
                       __fadd_rn(low, __fmul_rn(__fadd_rn(n, c.y), cs)));
}

// Evaluates one run: up to K words of 32 cells, word k at cells wd[k] of a node
// whose first cell is (nx, ny, nz)[k / 2]. Returns the words' leaf masks.
template <int K>
__device__ __forceinline__ void leaf_run(const LevelTree& T, const LeafTape& tp, uint4* stage, uint32_t slot_base,
                                         uint32_t lane,
                                         const float (&nx)[K / 2], const float (&ny)[K / 2], const float (&nz)[K / 2],
                                         const uint32_t (&wd)[K], uint32_t (&leaf)[K]) {
    const uint32_t lane_base = slot_base + lane * (4u * K);
    // (voxelizer/main.comp:74-79; the sums are whole numbers below 2^24, exact)
    FK<K> px, py, pz;
#pragma unroll
    for (int k = 0; k < K; k += 2) {
        float2 cx, cy, cz;
        if (T.dim == 4) {  // words 0 and 1
            cx.x = (float)(lane >> 4);
            cx.y = cx.x + 2.0f;
            cy.x = cy.y = (float)((lane >> 2) & 3u);
            cz.x = cz.y = (float)(lane & 3u);
        } else {
            uint32_t x, y, z;
            cell_xyz(wd[k] * 32u + lane, T.dim, T.dim_sh, &x, &y, &z);
            cx.x = (float)x;
            cy.x = (float)y;
            cz.x = (float)z;
            cell_xyz(wd[k + 1] * 32u + lane, T.dim, T.dim_sh, &x, &y, &z);
            cx.y = (float)x;
            cy.y = (float)y;
            cz.y = (float)z;
        }
        const float2 x = cell_low(nx[k / 2], cx, T.lx, T.cs), y = cell_low(ny[k / 2], cy, T.ly, T.cs),
                     z = cell_low(nz[k / 2], cz, T.lz, T.cs);
        px.v[k] = x.x;
        px.v[k + 1] = x.y;
        py.v[k] = y.x;
        py.v[k + 1] = y.y;
        pz.v[k] = z.x;
        pz.v[k + 1] = z.y;
    }
    // the inputs that are read as rows (rows 0 .. in slot order)
    uint32_t off = lane_base;
    if (tp.mask & 1u) {
        sts_k<K>(off, px);
        off += tp.stride;
    }
    if (tp.mask & 2u) {
        sts_k<K>(off, py);
        off += tp.stride;
    }
    if (tp.mask & 4u) {
        sts_k<K>(off, pz);
        off += tp.stride;
    }
    FK<K> r;
    if (tp.mask & 8u) {
#pragma unroll
        for (int k = 0; k < K; k++) r.v[k] = T.tt;
        sts_k<K>(off, r);
    }
#pragma unroll
    for (int k = 0; k < K; k++) r.v[k] = 0.0f;
    uint32_t at = 0;
    do {
        at = tp.ops > LEAF_OPS ? leaf_stage(tp, stage, at, lane) : tp.ops;
        leaf_exec<K>(smem_addr(stage), lane_base, r);
    } while (at < tp.ops);
    // the last instruction writes slot 0 (checked when a tape is made; kept by
    // shortening), so r is the result
#pragma unroll
    for (int k = 0; k < K; k++) leaf[k] = __ballot_sync(0xFFFFFFFFu, r.v[k] < 0.0f);
}

// Takes the next items: up to `most`, fewer as the rest gets small against the
// grid (a third of its share), so that the warps end together. Returns their
// number, 0 at the end.
__device__ __forceinline__ uint32_t leaf_fetch(unsigned long long* cursor, unsigned long long total, uint32_t warps,
                                               uint32_t most, uint32_t lane, unsigned long long* first) {
    unsigned long long f = 0;
    uint32_t c = 0;
    if (lane == 0) {
        const unsigned long long at = *reinterpret_cast<volatile unsigned long long*>(cursor);
        const unsigned long long left = at < total ? total - at : 0ull;
        c = (uint32_t)max(1ull, min((unsigned long long)most, left / (3ull * warps)));
        f = atomicAdd(cursor, (unsigned long long)c);
    }
    f = __shfl_sync(0xFFFFFFFFu, f, 0);
    c = __shfl_sync(0xFFFFFFFFu, c, 0);
    *first = f;
    return f < total ? (uint32_t)min((unsigned long long)c, total - f) : 0u;
}

template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 4 ? 5 : 20)
leaf_level_kernel(LevelLaunch p) {
    extern __shared__ __align__(16) unsigned char smem[];
    if (__ldcg(&p.cursor[1]) == 0ull) return;  // (point_level_kernel's launch)
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* wbase = smem + (size_t)warp * p.smem_per_warp;
    const uint32_t slot_bytes = p.smem_per_warp - LEAF_FIXED_BYTES;
    const uint32_t slot_base = smem_addr(wbase);
    uint4* stage = reinterpret_cast<uint4*>(wbase + slot_bytes);
    uint32_t* jobs = reinterpret_cast<uint32_t*>(stage + LEAF_OPS + 1);

    const uint32_t L = p.level, warps = gridDim.x * WARPS;
    const unsigned long long total = __ldcg(&p.prefix[p.n_trees]);
    // this warp's share of the scratch, 8-byte micro-ops (every tape fits: launch_level)
    const uint32_t cap = p.leaf_share;
    uint64_t* const scratch = reinterpret_cast<uint64_t*>(p.keep_scratch) + (size_t)(blockIdx.x * WARPS + warp) * cap;
    unsigned long long stat_work = 0;  // per lane
    LevelTree T{};
    unsigned long long t_lo = 0, t_hi = 0;
    bool have_tree = false;
    auto flush = [&]() {
        for (int off = 16; off > 0; off >>= 1) stat_work += __shfl_down_sync(0xFFFFFFFFu, stat_work, off);
        if (lane == 0 && stat_work) atomicAdd(&T.H->cell_instr[L], stat_work);
        stat_work = 0;
    };

    unsigned long long first;
    uint32_t got;
    while ((got = leaf_fetch(p.cursor, total, warps, p.leaf_chunk, lane, &first)) != 0) {
        for (uint32_t done = 0; done < got;) {
            const unsigned long long item = first + done;
            if (!have_tree || item >= t_hi) {
                if (have_tree) flush();
                const uint32_t ti = find_tree(p.prefix, p.n_trees, item);
                t_lo = __ldcg(&p.prefix[ti]);
                t_hi = __ldcg(&p.prefix[ti + 1]);
                T = load_tree(p.trees[ti], L, true);
                have_tree = true;
            }
            const uint32_t cnt = (uint32_t)min((unsigned long long)(got - done), t_hi - item);
            done += cnt;
            const uint32_t dim = T.dim, words = dim * dim * dim / 32;  // (a power of two)
            const bool small = dim == 4;
            const uint32_t unit_sh = small ? 0u : 3u * T.dim_sh - 8u;
            // item i: its node and, in larger nodes, which 8 words
            auto item_node = [&](uint32_t i, uint32_t* unit) {
                const unsigned long long local = item - t_lo + i;
                *unit = (uint32_t)local & ((1u << unit_sh) - 1u);
                const uint32_t node = (uint32_t)(local >> unit_sh);
                return p.eval_list ? __ldcg(&p.eval_list[node]) : node;  // (the others are copies)
            };
            auto record_of = [&](uint32_t node) { return T.nodes + T.ofs_l + (size_t)node * T.node_size; };

            // the distinct tapes of each 32 items, in the order of their first item
            uint32_t n_jobs = 0;
            __syncwarp();
#pragma unroll 1
            for (uint32_t q = 0; q < cnt; q += 32) {
                const bool valid = q + lane < cnt;
                uint32_t unit;
                const uint32_t tape = __ldcg(record_of(item_node(valid ? q + lane : q, &unit)));
                const uint32_t same = __match_any_sync(0xFFFFFFFFu, valid ? tape : ~0u);
                const uint32_t lead = __ballot_sync(0xFFFFFFFFu, valid && (same & lanemask_lt()) == 0u);
                if ((lead >> lane) & 1u) jobs[n_jobs + __popc(lead & lanemask_lt())] = tape;
                n_jobs += __popc(lead);
            }
            __syncwarp();

            uint32_t job = 0, job_lo = 0, job_hi = 0;         // the next job; those decoded: [job_lo, job_hi)
            uint32_t my_ofs = 0, my_ops = 0, my_rows = 0, my_n = 0;  // lane l: job job_lo + l
#pragma unroll 1
            for (uint32_t q = 0; q < cnt; q += 32) {
                uint32_t unit;
                const uint32_t node = item_node(q + lane < cnt ? q + lane : q, &unit);
                uint32_t* rec = record_of(node);
                const uint4 hd = __ldcg(reinterpret_cast<const uint4*>(rec));
                const float fx = (float)(hd.y * dim), fy = (float)(hd.z * dim), fz = (float)(hd.w * dim);
                uint32_t pend = __ballot_sync(0xFFFFFFFFu, q + lane < cnt);
#pragma unroll 1
                for (; pend; job++) {
                    if (job == job_hi) {
                        // decode the next jobs: as many as there are lanes and room
                        const uint64_t* r = job + lane < n_jobs ? T.tapes + jobs[job + lane] : nullptr;
                        my_n = r ? (uint32_t)__ldcg(r) : 0u;
                        uint32_t incl = (my_n + 1u) & ~1u;
                        for (int o = 1; o < 32; o <<= 1) {
                            const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                            if ((int)lane >= o) incl = min(incl + v, 1u << 30);
                        }
                        const bool fits = r && incl <= cap;
                        my_ofs = incl - ((my_n + 1u) & ~1u);
                        job_lo = job;
                        job_hi = job + __popc(__ballot_sync(0xFFFFFFFFu, fits));
                        __syncwarp();
                        if (job_hi - job >= LEAF_SERIAL) {
                            my_ops = leaf_decode(fits ? r : nullptr, scratch + my_ofs, slot_base + lane * 4u, &my_rows);
                        } else {
#pragma unroll 1
                            for (uint32_t j = 0; j < job_hi - job; j++) {
                                const uint2 m = leaf_decode_one(T.tapes + jobs[job + j], __shfl_sync(0xFFFFFFFFu, my_n, j),
                                                                scratch + __shfl_sync(0xFFFFFFFFu, my_ofs, j), lane);
                                if (lane == j) {
                                    my_ops = m.x;
                                    my_rows = m.y;
                                }
                            }
                        }
                        __syncwarp();
                    }
                    const int src_job = (int)(job - job_lo);
                    uint32_t members = __ballot_sync(0xFFFFFFFFu, hd.x == jobs[job]) & pend;
                    pend &= ~members;
                    LeafTape tp;
                    tp.saved = scratch + __shfl_sync(0xFFFFFFFFu, my_ofs, src_job);
                    tp.ops = __shfl_sync(0xFFFFFFFFu, my_ops, src_job);
                    tp.mask = __shfl_sync(0xFFFFFFFFu, my_rows, src_job);
                    tp.stride = (uint32_t)__popc(tp.mask) * 512u <= slot_bytes ? 512u : 256u;
                    const uint32_t n = __shfl_sync(0xFFFFFFFFu, my_n, src_job);
                    if (tp.ops <= LEAF_OPS) leaf_stage(tp, stage, 0, lane);
                    if ((members >> lane) & 1u)
                        stat_work += (unsigned long long)(small ? 64u : 256u) * n;

                    // the members' runs: dim-4 nodes in pairs, larger nodes' items 4
                    // words at a time (2 cells per lane where the rows are too many)
                    uint32_t at = 0;  // words of the first member's item that are done
                    auto run = [&](auto kc) {
                        constexpr int K = decltype(kc)::value;
                        uint32_t s[K / 2], wd[K], leaf[K], w = 0;
                        float nx[K / 2], ny[K / 2], nz[K / 2];
                        if (small) {
#pragma unroll
                            for (int m = 0; m < K / 2; m++) {  // (past the last member: it again)
                                s[m] = members ? (uint32_t)__ffs(members) - 1u : s[m ? m - 1 : 0];
                                members &= members - 1;
                                wd[2 * m] = 0;
                                wd[2 * m + 1] = 1;
                            }
                        } else {
                            const uint32_t src = (uint32_t)__ffs(members) - 1u;
                            w = 8u * __shfl_sync(0xFFFFFFFFu, unit, src) + at;
                            at += K;
                            if (at >= 8u) {
                                members &= members - 1;
                                at = 0;
                            }
#pragma unroll
                            for (int m = 0; m < K / 2; m++) s[m] = src;
#pragma unroll
                            for (int k = 0; k < K; k++) wd[k] = w + k;
                        }
#pragma unroll
                        for (int m = 0; m < K / 2; m++) {
                            nx[m] = __shfl_sync(0xFFFFFFFFu, fx, s[m]);
                            ny[m] = __shfl_sync(0xFFFFFFFFu, fy, s[m]);
                            nz[m] = __shfl_sync(0xFFFFFFFFu, fz, s[m]);
                        }
                        leaf_run<K>(T, tp, stage, slot_base, lane, nx, ny, nz, wd, leaf);
                        if (small) {
#pragma unroll
                            for (int m = 0; m < K / 2; m++)
                                if (lane == s[m])
                                    *reinterpret_cast<uint4*>(rec + 4) = make_uint4(leaf[2 * m], leaf[2 * m + 1], 0u, 0u);
                        } else {
                            uint32_t* o = record_of(__shfl_sync(0xFFFFFFFFu, node, s[0])) + 4;
                            uint32_t mine = 0;
#pragma unroll
                            for (int k = 0; k < K; k++)
                                if (lane == (uint32_t)k) mine = leaf[k];
                            if (lane < (uint32_t)K) {
                                o[w + lane] = mine;
                                o[words + w + lane] = 0u;  // the unused second mask word range
                            }
                        }
                    };
                    while (members) {
                        if (tp.stride == 512u) run(std::integral_constant<int, 4>{});
                        else run(std::integral_constant<int, 2>{});
                    }
                }
            }
        }
    }
    if (have_tree) flush();
}
