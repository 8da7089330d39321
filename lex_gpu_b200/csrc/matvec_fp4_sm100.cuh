// gemm_fp4 for m <= 16 (decode and speculative-verify steps): a split-K matvec that reads the
// packed weights from HBM once.
//
// Same operator as gemm_fp4_sm100.cuh (crates/lex-front/lx/gemm_fp4.lx:16-36): f16 x,
// weights decoded bit-exactly to f16, f32 accumulation.  The reference runs small m
// through different kernels with different arithmetic (crates/lex-msl/src/int8.rs:121-223
// quantises x to int16; crates/lex-front/src/llama.rs:444-499 keeps weights in f32); this
// one keeps gemm_fp4's semantics so one oracle covers every m.
//
// K is summed in 8 parts, slices of 128 columns dealt out in turns (part p: slices p, p + 8, ...), a warp each; a k of 4
// slices or fewer in 4, 2 or 1.  A block of 8 warps has all parts of 16 rows at a time, so that it reads 512 contiguous
// bytes of each row per round; or a cluster of 2, 4 or 8 blocks shares the parts, each block with as many more row blocks,
// and adds them up through distributed shared memory, always in the order of the parts.  What the cluster divides is the
// staged x: m = 4 at k = 17408 is 157 KB of it, one block an SM with x read twice over by each; divided by 8, four blocks of
// 4 warps or two of 8 (5120x17408 on a B200: 57.4 -> 22.1 us, back to back with other weights each time; W alone takes 7.7
// at the copy rate).
// Inside a slice, lane (g = lane/4, t = lane%4) owns rows g and g+8 and the two groups of 16
// columns 32t..32t+31: one 16-byte load of codes per row, two scale bytes, the factors of two
// groups per row.  The multiply-accumulate runs on the tensor cores (mma.sync m16n8k16,
// weights as the 16-row operand, up to 8 tokens as the 8-column operand): the integer and FP16
// pipes are taken by the decode, and the f16 x f16 products are exact in f32 either way.
// Because a contraction may visit K in any order, the 16 K-slots of one mma are mapped to
// 4 columns from each of the 4 lanes' own groups - no weight ever crosses lanes.
//
// Blocks are persistent when their x fits in shared memory (the usual case): x is staged once and
// the block walks over row blocks blockIdx.x, +gridDim.x, ...; the loads of the next slice -
// of the next row block at the end - are always in flight while a slice is decoded.
// x in shared memory: each 64-byte run (32 columns, what one lane consumes per slice) is
// stored 72 bytes apart and the token pitch is 32 (mod 128) bytes, which makes the quad's
// four 8-byte reads per token and the eight tokens of a warp hit distinct banks.
#pragma once
#include "sm100_ptx.cuh"
#include "fp4_decode.cuh"

namespace lexb {

constexpr uint32_t MV_ROWS = 16;
constexpr uint32_t MV_WARPS = 8;
constexpr uint32_t MV_THREADS = MV_WARPS * 32;
constexpr uint32_t MV_SLICE = 128;                   // K columns per warp iteration
constexpr uint32_t MV_ROUND = MV_SLICE * MV_WARPS;   // K columns per block round
constexpr uint32_t MV_PARTS = MV_WARPS;              // parts of K: part p is slices p, p + 8, ...
// one warp's sums of a row block: [16 tokens][MV_RED_PITCH], rows innermost (the pitch keeps a warp's stores off one bank)
constexpr uint32_t MV_RED_PITCH = 20;
__host__ __device__ constexpr uint32_t matvec_red_floats(uint32_t m) { return (m <= 8u ? 8u : 16u) * MV_RED_PITCH; }
// The packed weights come through a ring in shared memory filled by asynchronous copies (cp.async): a warp keeps
// MV_DEPTH slices in flight, each lane copying exactly the 2 x 16 bytes of codes it will decode itself (so the ring
// is a per-lane FIFO and its reads are conflict-free) and two lanes of each quad the quad's 2 x 8 scale bytes.
// With the loads in registers one slice ahead, the warps spent most of their time waiting for memory.
constexpr uint32_t MV_DEPTH = 3;
constexpr uint32_t MV_STAGE_BYTES = 2u * 512u + 128u;              // codes of row g, codes of row g + 8, scale bytes

struct MatvecArgs {
    const __half* x;      // [m, k]
    const uint8_t* wq;    // [n, k/2]
    const uint8_t* ws;    // [n, k/16]
    const float* wg;      // [n]
    const float* r;       // [m, n] or null
    float* y;             // [m, n]
    uint32_t m, n, k;
    uint32_t kc;          // K columns of x staged per chunk: multiple of MV_ROUND
    // powers of two, as their logarithms (a division by a run-time number costs a short launch more than its multiply)
    uint32_t log_cluster; // blocks that share the parts of K: 1, 2, 4 or 8
    uint32_t log_parts;   // parts that K has: 8, or 4, 2, 1 if that is as many as it has slices
    uint32_t log_group;   // row blocks a cluster works on at once: its warps / parts
    uint32_t log_tokens;  // tokens a block's warps stage at once: m rounded up, at most the block's warps
};

// token pitch in bytes: kc/32 runs of 72 bytes, padded to 32 (mod 128)
__host__ __device__ constexpr uint32_t matvec_x_pitch(uint32_t kc) {
    return (kc / 32u) * 72u + ((32u + 128u - ((kc / 32u) * 72u) % 128u) % 128u);
}
// two reduction buffers (alternating per row block), the ring (when used), then this block's share of the x chunk
__host__ __device__ constexpr uint32_t matvec_smem_bytes(uint32_t m, uint32_t kc, uint32_t warps, uint32_t cluster, bool ring) {
    return 2u * warps * matvec_red_floats(m) * 4u + (ring ? warps * MV_DEPTH * MV_STAGE_BYTES : 0u) + 128u + m * matvec_x_pitch(kc / cluster) + 16u;   // 128 bytes of zeros before x
}
__device__ __forceinline__ void mma_m16n8k16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct MvLoad {
    uint4 qa, qb;        // 32 codes of row g / row g+8
    uint32_t sa, sb;     // their two scale bytes (low 16 bits)
};

// 16, 8 or 0 bytes from global to shared memory without passing through registers; src_bytes = 0 fills with zeros
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_8(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <uint32_t N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// HI: m > 8, a second group of 8 tokens, whose staged x leaves no room for the ring: the weights come through registers,
// one slice ahead.  RAGGED: k % 128 != 0.
// WARPS: warps per SM the registers are cut to, 24 (80 registers a thread) or 16 (128).  With 16 the compiler overlaps the
// decode of one word with the next and with the multiply, which is worth more than the other warps (17408x5120, m = 1: 18.8 us
// with 16; 21.4 with 32, whose 64 registers spill) wherever the row blocks divide as well.  At 80 registers only the instance
// for m > 8 with a ragged k spills (20 bytes).
template <bool HI, bool RAGGED, uint32_t WARPS>
__global__ void __launch_bounds__(MV_THREADS, WARPS / MV_WARPS) matvec_fp4_kernel(const MatvecArgs a) {
    constexpr bool RING = !HI;
    constexpr uint32_t RED = matvec_red_floats(HI ? 16u : 8u);
    extern __shared__ __align__(16) uint8_t mv_smem[];
    const uint32_t tid = threadIdx.x, nthreads = blockDim.x, warps = nthreads >> 5, warp = tid >> 5, lane = tid & 31u;
    const uint32_t g = lane >> 2, t = lane & 3u;
    float* const red = reinterpret_cast<float*>(mv_smem);               // [2][warp][RED]
    uint8_t* const ring = mv_smem + 2u * warps * RED * 4u;              // [warp][MV_DEPTH] stages of packed weights
    uint8_t* const zeros = ring + (RING ? warps * MV_DEPTH * MV_STAGE_BYTES : 0u);   // 128 bytes: x of a token that does not exist
    uint8_t* const xs = zeros + 128u;
    const uint32_t lc = a.log_cluster, lp = a.log_parts, lr = a.log_group, lpp = lp - lc;
    const uint32_t C = 1u << lc, rank = C > 1u ? cluster_ctarank() : 0u;
    const uint32_t parts = 1u << lp, PP = 1u << lpp;                    // parts of K, of them in this block
    const uint32_t R = 1u << lr;                                        // row blocks the cluster works on at once: a group
    const uint32_t part = (rank << lpp) + (warp & (PP - 1u)), sub = warp >> lpp;     // this warp's part of K, and its row block of the group
    const uint32_t k = a.k, kc = a.kc;
    const uint32_t pitch = matvec_x_pitch(kc >> lc);
    const uint32_t slices = (k + MV_SLICE - 1u) / MV_SLICE;             // per row block
    const uint32_t row_blocks = a.n / MV_ROWS, groups = (row_blocks + R - 1u) >> lr;
    const uint32_t first_group = blockIdx.x >> lc, group_step = gridDim.x >> lc;
    const bool resident = kc >= k;                                      // all of x staged once

    // Launched with programmatic stream serialization: the blocks are in place when the launch ahead ends.  The next launch's
    // blocks are let in only then.  Let in earlier, they gather, as many as fit, on the SMs that this launch has left free, and
    // its own turn then waits for the fullest SM (1024x4096, m = 1, back to back: 5.1 us; 4.0 like this).
    grid_dependency_wait();
    allow_dependents();

    // lanes whose token does not exist (and lanes past the end of K) read the zero block instead
    const bool have_lo = g < a.m, have_hi = HI && (g + 8u) < a.m;

    // this block's parts of x[:, k0:k1] -> shared memory, asynchronously and 8 bytes at a time (coalesced in,
    // conflict-free out): slice s of the chunk is the block's slice (s / 8) * PP + s % PP.  A warp takes a token's slice at a
    // time, 256 bytes; the warps are dealt to the tokens, and within a token to its slices.
    auto stage_x = [&](uint32_t k0, uint32_t k1) {
        const uint32_t sc = (k1 - k0 + MV_SLICE - 1u) / MV_SLICE, rem = sc & (parts - 1u), p0 = rank << lpp;
        const uint32_t mine = ((sc >> lp) << lpp) + (rem <= p0 ? 0u : (rem - p0 < PP ? rem - p0 : PP));
        const uint32_t lt = a.log_tokens, per_token = warps >> lt;
        for (uint32_t tok = warp & ((1u << lt) - 1u); tok < a.m; tok += 1u << lt) {
            const __half* src = a.x + (size_t)tok * k + k0;
            const uint32_t dst = smem_u32(xs) + tok * pitch + (lane >> 3) * 72u + (lane & 7u) * 8u;
            for (uint32_t j = warp >> lt; j < mine; j += per_token) {
                const uint32_t col = (((j >> lpp) << lp) + p0 + (j & (PP - 1u))) * MV_SLICE + 4u * lane;
                if (!RAGGED || k0 + col < k1) cp_async_8(dst + j * 288u, src + col, 8u);
            }
        }
        if (tid < 16u) *reinterpret_cast<uint2*>(zeros + tid * 8u) = make_uint2(0u, 0u);
    };

    // This warp's slices of a row block: part, part + 8, ... (fewer parts: one slice, or none)
    const uint32_t my_slices = part < slices ? (slices - part + parts - 1u) >> lp : 0u;
    const size_t q_row = k / 2u, s_row = k / 16u, q_pitch8 = 8u * q_row;
    // The copy cursor: this lane's codes of the next slice to be asked for (row g; row g + 8 is q_pitch8 further) and its
    // scale bytes - in the ring lanes t = 0 and 1 of a quad copy the quad's 8 of row g and of row g + 8.
    const uint8_t *q_next = nullptr, *s_next = nullptr;
    uint32_t rb_c = first_group * R + sub, left_c = 0;
    auto cursor_to = [&](uint32_t rb) {
        const size_t row = (size_t)rb * MV_ROWS + g;
        q_next = a.wq + row * q_row + part * (MV_SLICE / 2u) + 16u * t;
        s_next = a.ws + (row + (RING && !RAGGED ? 8u * (t & 1u) : 0u)) * s_row + part * (MV_SLICE / 16u) + (RING && !RAGGED ? 0u : 2u * t);
        left_c = my_slices;
    };
    auto cursor_step = [&]() {
        q_next += MV_ROUND / 2u;
        s_next += MV_ROUND / 16u;
        if (--left_c == 0u) {
            rb_c += group_step * R;
            cursor_to(rb_c);
        }
    };
    // (k % 32 == 0: a lane's 32 columns of a slice are in K together or not at all)
    auto cursor_in_k = [&]() { return !RAGGED || (part + (my_slices - left_c) * parts) * MV_SLICE + 32u * t < k; };
    cursor_to(rb_c);

    // This warp's ring.  Stage layout: [codes of row g: 32 lanes x 16 B][codes of row g + 8][scales: 16 rows x 8 B].
    uint8_t* const my_ring = ring + warp * (MV_DEPTH * MV_STAGE_BYTES);
    uint32_t st_c = 0, st = 0;                                          // byte offsets of the stages: next to fill, next to use
    // asynchronous copies of the next slice (a commit group of its own, also when there is none: the groups are counted)
    uint32_t scales = 0, scales_b = 0, scales_at = 0;                   // (RAGGED) loaded scale bytes and the stage they belong to
    auto issue_copies = [&]() {
        if (RAGGED) {
            uint8_t* sdst = my_ring + scales_at + 1024u + g * 8u + 2u * t;
            *reinterpret_cast<unsigned short*>(sdst) = static_cast<unsigned short>(scales);
            *reinterpret_cast<unsigned short*>(sdst + 64u) = static_cast<unsigned short>(scales_b);
        }
        if (rb_c < row_blocks && my_slices != 0u) {
            const uint32_t in_k = cursor_in_k() ? 1u : 0u;              // zeros past the end of K
            const uint32_t dst = smem_u32(my_ring) + st_c + lane * 16u;
            cp_async_16(dst, in_k ? q_next : a.wq, 16u * in_k);
            cp_async_16(dst + 512u, in_k ? q_next + q_pitch8 : a.wq, 16u * in_k);
            if (RAGGED) {
                // k % 128 != 0: a row's scale bytes are not 8-byte aligned, so each lane loads its own two of both rows
                // and stores them when the next slice is asked for, not waiting for them here
                scales = in_k ? __ldg(reinterpret_cast<const unsigned short*>(s_next)) : 0u;
                scales_b = in_k ? __ldg(reinterpret_cast<const unsigned short*>(s_next + 8u * s_row)) : 0u;
                scales_at = st_c;
            } else if (t < 2u) {
                cp_async_8(smem_u32(my_ring) + st_c + 1024u + (g + 8u * t) * 8u, s_next, 8u);
            }
            cursor_step();
        }
        st_c = st_c == (MV_DEPTH - 1u) * MV_STAGE_BYTES ? 0u : st_c + MV_STAGE_BYTES;
    };
    auto issue_next = [&]() {
        issue_copies();
        cp_async_commit();
    };
    // the register path (RING = false): this lane's loads for the next slice
    auto load_next = [&]() {
        MvLoad L{};                                                     // past the end: zero codes (their lane multiplies by 1.0)
        if (rb_c < row_blocks && my_slices != 0u) {
            if (cursor_in_k()) {
                L.qa = __ldg(reinterpret_cast<const uint4*>(q_next));
                L.qb = __ldg(reinterpret_cast<const uint4*>(q_next + q_pitch8));
                L.sa = __ldg(reinterpret_cast<const unsigned short*>(s_next));
                L.sb = __ldg(reinterpret_cast<const unsigned short*>(s_next + 8u * s_row));
            }
            cursor_step();
        }
        return L;
    };
    auto take = [&]() {
        MvLoad L;
        const uint8_t* sp = my_ring + st;
        L.qa = *reinterpret_cast<const uint4*>(sp + lane * 16u);
        L.qb = *reinterpret_cast<const uint4*>(sp + 512u + lane * 16u);
        L.sa = *reinterpret_cast<const unsigned short*>(sp + 1024u + g * 8u + 2u * t);
        L.sb = *reinterpret_cast<const unsigned short*>(sp + 1024u + 64u + g * 8u + 2u * t);
        st = st == (MV_DEPTH - 1u) * MV_STAGE_BYTES ? 0u : st + MV_STAGE_BYTES;
        return L;
    };

    float wg_a = 0.0f, wg_b = 0.0f;                                     // row scales of the warp's next row block
    auto load_row_scales = [&](uint32_t rb) {
        if (rb < row_blocks) {
            wg_a = __ldg(a.wg + rb * MV_ROWS + g);
            wg_b = __ldg(a.wg + rb * MV_ROWS + g + 8u);
        }
    };
    load_row_scales(rb_c);

    // The first weights go out before x (they come from HBM, x mostly from L2) and are waited for with it.  The copies run
    // MV_DEPTH slices ahead of the decode, in the same order: this warp's slices of a row block, then those of its next one.
    MvLoad nxt{};
    if constexpr (RING) issue_copies();
    else nxt = load_next();
    if (resident) stage_x(0, k);
    cp_async_commit();
    if constexpr (RING) {
#pragma unroll
        for (uint32_t d = 1; d < MV_DEPTH; d++) issue_next();
    }
    // (the row scales are on their way since before the copies: what follows from them is worked out under the wait)
    RowScale ga = make_row_scale(wg_a), gb = make_row_scale(wg_b);
    if (resident) {
        cp_async_wait<RING ? MV_DEPTH - 1u : 0u>();
        __syncthreads();
    }

    uint32_t parity = 0;
    // this lane's 64 bytes of x per token and slice: runs of 72 bytes, 4 per slice of the block
    const uint32_t x_own = (warp & (PP - 1u)) * 288u + t * 72u, x_step = PP * 288u;

    for (uint32_t grp_i = first_group; grp_i < groups; grp_i += group_step, parity ^= 1u) {
        const uint32_t rb = grp_i * R + sub;                            // (>= row_blocks in the last group: this warp has no rows)
        const bool have_rb = rb < row_blocks;
        load_row_scales(rb + group_step * R);                           // (in flight during this row block)
        // rows g and g + 8 are decoded side by side: their scale bytes share a word, g's in the low half
        const uint32_t below = prmt(ga.below, gb.below, 0x5410u), above = prmt(ga.above, gb.above, 0x5410u);
        float c_lo[4] = {0.f, 0.f, 0.f, 0.f};
        float c_hi[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t left = have_rb ? my_slices : 0u;

        for (uint32_t k0 = 0; k0 < k; k0 += kc) {
            uint32_t here = left;                                       // of them in this chunk
            if (!resident) {
                const uint32_t k1 = (k0 + kc < k) ? (k0 + kc) : k;
                __syncthreads();                                        // previous chunk fully consumed
                stage_x(k0, k1);
                cp_async_commit();
                cp_async_wait<0>();
                __syncthreads();
                here = min(left, kc / MV_ROUND);                        // (all chunks but the last are whole rounds)
            }
            left -= here;
            const uint8_t* x_lo = have_lo ? xs + g * pitch + x_own : zeros;
            const uint8_t* x_hi = have_hi ? xs + (g + 8u) * pitch + x_own : zeros;
            const uint32_t lo_step = have_lo ? x_step : 0u, hi_step = have_hi ? x_step : 0u;
            uint32_t col = k0 + part * MV_SLICE + 32u * t;              // (RAGGED)
            for (; here != 0u; here--, x_lo += lo_step, x_hi += hi_step, col += MV_ROUND) {
                MvLoad cur;
                if constexpr (RING) {
                    cp_async_wait<MV_DEPTH - 1>();                      // the oldest slice in flight has landed
                    __syncwarp();                                       // (the scale bytes were copied by two lanes of the quad)
                    cur = take();
                    __syncwarp();                                       // every lane has read the stage: refill it
                    issue_next();
                } else {
                    cur = nxt;
                    nxt = load_next();                                  // of this row block, or the first of the warp's next one
                }
                const bool in_range = !RAGGED || col < k;
                if (RAGGED && !in_range) x_lo = x_hi = zeros;           // (a part's last slice)
                // eight codes of row g and of row g + 8 (word wd of group grp of the slice), decoded, times x
                auto multiply = [&](uint32_t grp, uint32_t wd, const uint32_t (&oa)[4], const uint32_t (&ob)[4]) {
#pragma unroll
                    for (uint32_t hf = 0; hf < 2; hf++) {
                        const uint32_t unit = 4u * grp + 2u * wd + hf;   // 8-byte unit of the lane's 64 bytes
                        const uint2 bl = *reinterpret_cast<const uint2*>(x_lo + 8u * unit);
                        mma_m16n8k16(c_lo, oa[2 * hf], ob[2 * hf], oa[2 * hf + 1], ob[2 * hf + 1], bl.x, bl.y);
                        if (HI) {
                            const uint2 bh = *reinterpret_cast<const uint2*>(x_hi + 8u * unit);
                            mma_m16n8k16(c_hi, oa[2 * hf], ob[2 * hf], oa[2 * hf + 1], ob[2 * hf + 1], bh.x, bh.y);
                        }
                    }
                };
                auto word = [](const uint4& q, uint32_t grp, uint32_t wd) { return grp ? (wd ? q.w : q.z) : (wd ? q.y : q.x); };
                const uint32_t sc = prmt(cur.sa, cur.sb, 0x5410u);
                if (__all_sync(0xFFFFFFFFu, products_ok(sc, below, above))) {
                    const GroupFactors fa = group_factors(sc << 20, sc << 12, ga.up), fb = group_factors(sc << 4, sc >> 4, gb.up);
#pragma unroll
                    for (uint32_t grp = 0; grp < 2; grp++) {
                        const uint32_t base_a = grp ? high_half_twice(fa.base) : low_half_twice(fa.base);
                        const uint32_t extra_a = grp ? high_half_twice(fa.extra) : low_half_twice(fa.extra);
                        const uint32_t base_b = grp ? high_half_twice(fb.base) : low_half_twice(fb.base);
                        const uint32_t extra_b = grp ? high_half_twice(fb.extra) : low_half_twice(fb.extra);
#pragma unroll
                        for (uint32_t wd = 0; wd < 2; wd++) {
                            uint32_t oa[4], ob[4];
                            multiply8(word(cur.qa, grp, wd), base_a, extra_a, oa[0], oa[1], oa[2], oa[3]);
                            multiply8(word(cur.qb, grp, wd), base_b, extra_b, ob[0], ob[1], ob[2], ob[3]);
                            multiply(grp, wd, oa, ob);
                        }
                    }
                } else {
                    // a lane past the end of K multiplies zero codes by 1.0, never by a row scale
                    // that might be infinite
                    const float ga_e = in_range ? ga.wg : 1.0f, gb_e = in_range ? gb.wg : 1.0f;
#pragma unroll
                    for (uint32_t grp = 0; grp < 2; grp++) {
                        const GroupTable ta = make_group_table(grp ? cur.sa >> 8 : cur.sa & 0xFFu, ga_e);
                        const GroupTable tb = make_group_table(grp ? cur.sb >> 8 : cur.sb & 0xFFu, gb_e);
#pragma unroll
                        for (uint32_t wd = 0; wd < 2; wd++) {
                            uint32_t oa[4], ob[4];
                            decode8(ta, word(cur.qa, grp, wd), oa[0], oa[1], oa[2], oa[3]);
                            decode8(tb, word(cur.qb, grp, wd), ob[0], ob[1], ob[2], ob[3]);
                            multiply(grp, wd, oa, ob);
                        }
                    }
                }
            }
        }

        // The 8 parts are added in the order of the parts, whichever blocks hold them, so a row's result depends neither
        // on the cluster nor on the batch.  Two buffers alternate, so one barrier per group is enough.
        float* const rw = red + (parity * warps + warp) * RED;
        if (2u * t < a.m) {
            rw[(2u * t) * MV_RED_PITCH + g] = c_lo[0];
            rw[(2u * t + 1u) * MV_RED_PITCH + g] = c_lo[1];
            rw[(2u * t) * MV_RED_PITCH + g + 8u] = c_lo[2];
            rw[(2u * t + 1u) * MV_RED_PITCH + g + 8u] = c_lo[3];
        }
        if (HI) {
            rw[(8u + 2u * t) * MV_RED_PITCH + g] = c_hi[0];
            rw[(9u + 2u * t) * MV_RED_PITCH + g] = c_hi[1];
            rw[(8u + 2u * t) * MV_RED_PITCH + g + 8u] = c_hi[2];
            rw[(9u + 2u * t) * MV_RED_PITCH + g + 8u] = c_hi[3];
        }
        if (C > 1u) cluster_sync_all();
        else __syncthreads();
        // outputs of the group: m tokens x R * 16 rows, four rows a thread, shared out over the cluster's threads
        const uint32_t log_quads = lr + 2u;
        for (uint32_t o_i = rank * nthreads + tid; o_i < (a.m << log_quads); o_i += nthreads << lc) {
            const uint32_t tok = o_i >> log_quads, ri = (o_i & ((1u << log_quads) - 1u)) * 4u;
            const uint32_t row = (grp_i << (lr + 4u)) + ri;
            if (row >= a.n) continue;
            const float* rp = red + (parity * warps + ((ri >> 4) << lpp)) * RED + tok * MV_RED_PITCH + (ri & 15u);
            float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
            auto add = [&](const float4& v) { s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; };
            if (C > 1u) {
                const uint32_t rp_u32 = smem_u32(rp);
#pragma unroll
                for (uint32_t p = 0; p < MV_PARTS; p++)
                    if (p < parts) add(ld_shared_cluster_f32x4(map_to_cta(rp_u32 + (p & (PP - 1u)) * (RED * 4u), p >> lpp)));
            } else {
#pragma unroll
                for (uint32_t p = 0; p < MV_PARTS; p++)
                    if (p < parts) add(*reinterpret_cast<const float4*>(rp + p * RED));
            }
            const size_t o = (size_t)tok * a.n + row;                       // (n % 16 == 0: rows of whole 16-byte quads)
            if (a.r) add(__ldg(reinterpret_cast<const float4*>(a.r + o)));
            *reinterpret_cast<float4*>(a.y + o) = s;
        }
        if (grp_i + group_step < groups) {
            ga = make_row_scale(wg_a);
            gb = make_row_scale(wg_b);
        }
    }
    if (C > 1u) cluster_sync_all();                                     // a block's sums are read by the others until here
}

}  // namespace lexb
