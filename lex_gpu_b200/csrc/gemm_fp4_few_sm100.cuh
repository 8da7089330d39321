// gemm_fp4 for few tokens (m <= 64) on sm_100a: the weights as one stream per SM.
//
// With few tokens a launch is its weights: bytes that come from HBM once, each of them decoded once, multiplied by next to
// nothing.  Whole tiles dealt out one per block leave SMs idle (224 tiles of n = 28672 on 148 SMs: two waves) and pay a
// block's set-up per tile.  Here there is one block per SM, and the packed weights - blocks of 128 rows x 256 columns of K -
// are numbered through the row tiles, K innermost: a cluster of C blocks has whole row tiles, and each of its blocks an
// equal, contiguous share of their blocks of weights, whatever tile boundaries it crosses.  The rings never drain at one.
//
// A block's share of a tile is a segment.  A tile that lies in one share is stored by that block; of a tile cut by a
// boundary every share leaves its sums in shared memory, and after the last segment - one barrier across the cluster - the
// blocks that have a part of it add the parts in the order of K, straight from one another's shared memory, and store y.
// Nothing of it passes through global memory, no block waits for another before that barrier, and a launch needs no
// workspace.  The cuts depend on n, k and the cluster; the cluster, the number of accumulators (8, 4 or 2) and the choice of this kernel
// depend on the number of tokens, so a token's last bits may depend on its batch, as in the two-CTA kernel's plans.
//
// Roles (736 threads): warps 0-15 decode - eight take the even blocks of weights, eight the odd ones, a warp 32 rows and two of
// the four K steps (64 columns each), a row a thread - into tensor memory, from where the MMAs take them as their A operand (M = 128 rows); warps
// 16-19 the epilogue of a segment during the next one's main loop; warp 20 the copies of the packed weights, 21 of x, 22
// the MMAs (N = 16, 32 or 64 tokens).
//
// What bounds it: the decode warps' turns, half decode (560 of 1450 clocks a K step when a turn was one K step) and half barriers,
// stores and fences; without the decode 28672 x 4096 took 21.6 us at 32 tokens, without the MMAs 29.3, with everything 32.0 and, with
// two K steps a turn, 29.4 in whole calls (the two-CTA kernel: 41.2; the bytes alone 10.7).  17408 x 5120 at 16 / 32 / 64 tokens: 18.9 /
// 19.4 / 20.7 us (64 by the two-CTA kernel: 24.9).
//
// Tensor memory: columns 0-255 two sets of accumulators (segments alternate), 128 columns each: 8, 4 or 2 accumulators of N
// columns that take the K steps in turn, so that each has an eighth, a quarter or half of the truncating additions; columns
// 256-511 the decoded weights, two blocks.
#pragma once
#include "fp4_decode.cuh"
#include "gemm_fp4_sm100.cuh"
#include "gemm_fp4_sm100_pair.cuh"
#include "sm100_ptx.cuh"

namespace lexb {

constexpr uint32_t FEW_ROWS = 128;
constexpr uint32_t FEW_K = PAIR_RAW_K;                 // columns of K per block of weights
constexpr uint32_t FEW_MAX_TOKENS = 64;
constexpr uint32_t FEW_DEQ_WARPS = 16;
constexpr uint32_t FEW_WARP_EPI = 16, FEW_WARP_RAW = 20, FEW_WARP_X = 21, FEW_WARP_MMA = 22;
constexpr uint32_t FEW_THREADS = 32u * 23u;
constexpr uint32_t FEW_MAX_CLUSTER = 8;
constexpr uint32_t FEW_ACC_SET = 128;                  // columns of one set of accumulators
constexpr uint32_t FEW_W_COL0 = 2u * FEW_ACC_SET;      // first column of the decoded weights
constexpr uint32_t FEW_W_SLOTS = 2;                    // blocks of them

struct FewArgs {
    const float* wg;         // [n]
    const float* r;          // [m, n] or null
    float* y;                // [m, n]
    uint16_t* act;           // gate/up fused: f16 [m, n / 2] instead of y
    uint32_t* status;
    uint32_t m, n, k;
    uint32_t cluster;        // blocks that share the tiles of a cluster
    uint32_t x_stages, raw_stages;
    uint32_t flags;          // bit 1: the packed weights are constant, copied and decoded ahead of the stream's order
};

// tokens of an MMA (N)
__host__ __device__ constexpr uint32_t few_cols(uint32_t m) { return m <= 16u ? 16u : m <= 32u ? 32u : 64u; }
__host__ __device__ constexpr uint32_t few_x_stage_bytes(uint32_t cols) { return cols * 128u * (FEW_K / GEMM_BK); }
// x ring, packed weights, the sums of a share's first segment, barriers, slot + flag, alignment slack
__host__ __device__ constexpr uint32_t few_smem_bytes(uint32_t m, uint32_t sx, uint32_t sr) {
    return sx * few_x_stage_bytes(few_cols(m)) + sr * PAIR_RAW_BYTES + m * FEW_ROWS * 4u + (2u * sx + 2u * sr + 2u * FEW_W_SLOTS + 4u) * 8u + 16u + 1024u;
}

template <uint32_t N>
__global__ void __launch_bounds__(FEW_THREADS, 1)
gemm_fp4_few_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_wq,
                    const __grid_constant__ CUtensorMap tmap_ws, const FewArgs a) {
    constexpr uint32_t ACCS = FEW_ACC_SET / N;           // accumulators of a set
    constexpr uint32_t STEPS = FEW_K / GEMM_BK;          // K steps per block of weights
    constexpr uint32_t XB = N * 128u, XSB = STEPS * XB;  // bytes of an x tile of one K step, of a stage
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t base = (raw_addr + 1023u) & ~1023u;
    uint8_t* const smem = smem_raw + (base - raw_addr);

    const uint32_t SX = a.x_stages, SR = a.raw_stages;
    const uint32_t raw_base = base + SX * XSB;
    const uint32_t head = raw_base + SR * PAIR_RAW_BYTES;                       // sums [m][128] of a share's first segment
    const uint32_t bars = head + a.m * FEW_ROWS * 4u;
    auto raw_full = [&](uint32_t s) { return bars + 8u * s; };
    auto raw_empty = [&](uint32_t s) { return bars + 8u * (SR + s); };
    auto x_full = [&](uint32_t s) { return bars + 8u * (2u * SR + s); };
    auto x_empty = [&](uint32_t s) { return bars + 8u * (2u * SR + SX + s); };
    const uint32_t wbars = bars + 8u * (2u * SR + 2u * SX);
    auto w_full = [&](uint32_t s) { return wbars + 8u * s; };
    auto w_empty = [&](uint32_t s) { return wbars + 8u * (FEW_W_SLOTS + s); };
    auto acc_full = [&](uint32_t set) { return wbars + 8u * (2u * FEW_W_SLOTS + set); };
    auto acc_empty = [&](uint32_t set) { return wbars + 8u * (2u * FEW_W_SLOTS + 2u + set); };
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(smem + (wbars - base) + (2u * FEW_W_SLOTS + 4u) * 8u);
    volatile uint32_t* const abort_flag = tmem_slot + 1;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    // This cluster's tiles, and this block's share [u0, u1) of their blocks of weights.
    const uint32_t C = a.cluster, rank = C > 1u ? cluster_ctarank() : 0u;
    const uint32_t clusters = gridDim.x / C, cid = blockIdx.x / C;
    const uint32_t tiles = a.n / FEW_ROWS, U = a.k / FEW_K;
    const uint32_t t_lo = cid * tiles / clusters, t_hi = (cid + 1u) * tiles / clusters;
    const uint32_t B = (t_hi - t_lo) * U;
    auto share = [&](uint32_t rk) { return rk * B / C; };
    const uint32_t u0 = share(rank), u1 = share(rank + 1u);
    const uint32_t tile0 = u0 / U, kb0 = u0 - tile0 * U;                         // (tile counted within the cluster)

    if (warp == FEW_WARP_RAW && lane == 0) {
        prefetch_tensormap(&tmap_wq);
        prefetch_tensormap(&tmap_ws);
    }
    if (warp == FEW_WARP_X && lane == 0) prefetch_tensormap(&tmap_x);
    if (warp == 0) {
        if (lane == 0) *abort_flag = 0;
        const uint32_t nbar = 2u * SR + 2u * SX + 2u * FEW_W_SLOTS + 4u, wb = 2u * SR + 2u * SX;
        for (uint32_t b = lane; b < nbar; b += 32u) {
            uint32_t count = 1;
            if (b >= SR && b < 2u * SR) count = FEW_DEQ_WARPS / FEW_W_SLOTS;         // raw_empty
            if (b >= wb && b < wb + FEW_W_SLOTS) count = FEW_DEQ_WARPS / FEW_W_SLOTS;      // w_full
            if (b >= wb + 2u * FEW_W_SLOTS + 2u) count = 4u;                         // acc_empty: the epilogue warps
            mbar_init(bars + 8u * b, count);
        }
        __syncwarp();
        fence_mbar_init();
    }
    if (warp == FEW_WARP_MMA) {
        tmem_alloc(smem_u32(tmem_slot), PAIR_TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    allow_dependents();                                                      // (not before this block holds its columns: see tmem_alloc)
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    // With constant weights their copies and decode start while the launch ahead still runs, and join the stream's order
    // before their first wait for a slot; everything else waits for it here.
    const bool early_w = (a.flags & 2u) != 0u;
    if (!(early_w && (warp == FEW_WARP_RAW || warp < FEW_DEQ_WARPS))) grid_dependency_wait();

    if (warp == FEW_WARP_RAW) {
        // ---------------------------------------------------------------- copies of the packed weights
        if (lane == 0) {
            RingPos pr;
            uint32_t kb = kb0, row = (t_lo + tile0) * FEW_ROWS;
            for (uint32_t u = u0; u < u1; u++, pr.advance(SR)) {
                if (early_w && u == u0 + SR) grid_dependency_wait();         // the ring is full: join the stream's order
                if (!mbar_wait(raw_empty(pr.s), pr.ph ^ 1u, abort_flag)) {
                    atomicOr(a.status, ST_WAIT_EMPTY_TMA);
                    *abort_flag = 1;
                    break;
                }
                mbar_arrive_expect_tx(raw_full(pr.s), PAIR_RAW_BYTES);
                const uint32_t dst = raw_base + pr.s * PAIR_RAW_BYTES;
                tma_load_2d(dst, &tmap_wq, (int)(kb * (FEW_K / 2u)), (int)row, raw_full(pr.s));
                tma_load_2d(dst + PAIR_RAW_WQ_BYTES, &tmap_ws, (int)(kb * (FEW_K / 16u)), (int)row, raw_full(pr.s));
                if (++kb == U) {
                    kb = 0;
                    row += FEW_ROWS;
                }
            }
            if (*abort_flag) {                                               // copies still in flight: a bounded time to land
                const long long t0 = clock64();
                while (clock64() - t0 < 400000) {
                }
            }
        }
        __syncwarp();
    } else if (warp == FEW_WARP_X) {
        // ---------------------------------------------------------------- copies of x
        if (lane == 0) {
            RingPos px;
            uint32_t kb = kb0;
            for (uint32_t u = u0; u < u1; u++, px.advance(SX)) {
                if (!mbar_wait(x_empty(px.s), px.ph ^ 1u, abort_flag)) {
                    atomicOr(a.status, ST_WAIT_EMPTY_TMA);
                    *abort_flag = 1;
                    break;
                }
                mbar_arrive_expect_tx(x_full(px.s), STEPS * a.m * 128u);     // (rows past m keep what they hold: columns nobody reads)
#pragma unroll
                for (uint32_t i = 0; i < STEPS; i++)
                    tma_load_2d(base + px.s * XSB + i * XB, &tmap_x, (int)(kb * FEW_K + i * GEMM_BK), 0, x_full(px.s));
                if (++kb == U) kb = 0;
            }
            if (*abort_flag) {
                const long long t0 = clock64();
                while (clock64() - t0 < 400000) {
                }
            }
        }
        __syncwarp();
    } else if (warp == FEW_WARP_MMA) {
        // ---------------------------------------------------------------- MMAs: the whole warp in the loop, one lane issues
        const uint32_t idesc = umma_idesc_f16_f32(128u, N);
        const uint32_t x_lo0 = umma_desc_lo(base);
        RingPos px, pw;
        uint32_t kb = kb0, seg = 0, step = 0;                                // step: K steps of the segment so far
        for (uint32_t u = u0; u < u1; u++, px.advance(SX), pw.advance(FEW_W_SLOTS)) {
            const uint32_t set = seg & 1u;
            bool ok = true;
            if (step == 0u && seg >= 2u) ok = mbar_wait(acc_empty(set), ((seg >> 1) - 1u) & 1u, abort_flag);
            ok = ok && mbar_wait(x_full(px.s), px.ph, abort_flag) && mbar_wait(w_full(pw.s), pw.ph, abort_flag);
            if (!__all_sync(0xFFFFFFFFu, ok)) {
                atomicOr(a.status, ST_WAIT_X_FULL | ST_WAIT_W_FULL);
                *abort_flag = 1;
                break;
            }
            tc_fence_after_sync();
            const uint32_t d = tmem_base + set * FEW_ACC_SET, at = tmem_base + FEW_W_COL0 + pw.s * (STEPS * 32u);
            const uint32_t xt = x_lo0 + px.s * (XSB >> 4);
            const bool last = kb + 1u == U || u + 1u == u1;
            if (elect_one()) {
#pragma unroll
                for (uint32_t i = 0; i < STEPS; i++) {
                    const uint32_t acc = d + ((step + i) % ACCS) * N;
#pragma unroll
                    for (uint32_t kk = 0; kk < GEMM_BK / 16u; kk++)
                        umma1_ts_flag(acc, at + 32u * i + 8u * kk, xt + i * (XB >> 4) + 2u * kk, idesc, (step + i >= ACCS || kk > 0u) ? 1u : 0u);
                }
                umma_commit(w_empty(pw.s));
                umma_commit(x_empty(px.s));
                if (last) umma_commit(acc_full(set));
            }
            __syncwarp();
            step += STEPS;
            if (++kb == U) kb = 0;
            if (last) {
                step = 0;
                seg++;
            }
        }
        __syncwarp();
    } else if (warp < FEW_DEQ_WARPS) {
        // ---------------------------------------------------------------- decode: half of every second block of weights, a row a thread
        // Two sets of eight warps take the even and the odd blocks, each into a slot of its own; a warp has 32 rows and two of
        // the four K steps, so that its waits, fences and arrivals - as long as the decode of a K step even where nothing is
        // waited for - come once per two K steps.  (Its parity waits are right although it passes over every second block: before it
        // stored the block before, the MMAs of the one before that were complete, so no barrier is two phases behind the one
        // awaited as long as the ring of packed blocks has four.)
        const uint32_t set = warp >> 3, half = (warp >> 2) & 1u, r = 32u * (warp & 3u) + lane;
        const uint32_t sw_xor = r & 7u;
        const uint8_t* const raw0 = smem + (raw_base - base) + r * 128u;
        const uint32_t sc_off = PAIR_RAW_WQ_BYTES - r * 128u + r * 16u + 8u * half;
        const uint32_t dst = tmem_base + ((32u * (warp & 3u)) << 16) + FEW_W_COL0 + set * (STEPS * 32u) + 64u * half;
        uint32_t kb = kb0 + set, tile = t_lo + tile0;
        auto load_wg = [&](uint32_t t) { return t < tiles ? __ldg(a.wg + (size_t)t * FEW_ROWS + r) : 0.0f; };
        float wg_now = load_wg(tile), wg_next = load_wg(tile + 1u);
        RowScale g = make_row_scale(wg_now);
        uint32_t turn = 0;                                                   // phase of this set's slot
        RingPos pr;
        pr.advance_by(set, SR);
        for (uint32_t u = u0 + set; u < u1; u += FEW_W_SLOTS, kb += FEW_W_SLOTS, pr.advance_by(FEW_W_SLOTS, SR), turn ^= 1u) {
            if (kb >= U) {                                                   // on to the tile that block is in
                uint32_t over = 0;
                do {
                    kb -= U;
                    over++;
                } while (kb >= U);
                tile += over;
                g = make_row_scale(over == 1u ? wg_next : load_wg(tile));
                wg_next = load_wg(tile + 1u);
            }
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(raw_full(pr.s), pr.ph, abort_flag))) {
                atomicOr(a.status, ST_WAIT_X_FULL);
                *abort_flag = 1;
                break;
            }
            const uint8_t* const raw = raw0 + pr.s * PAIR_RAW_BYTES;
            const uint2 sc = *reinterpret_cast<const uint2*>(raw + sc_off);
            bool ok = true;
#pragma unroll
            for (uint32_t i = 0; i < 2; i++) {
                const uint32_t q = 2u * half + i;
                const uint4 c0 = *reinterpret_cast<const uint4*>(raw + (((2u * q) ^ sw_xor) << 4));
                const uint4 c1 = *reinterpret_cast<const uint4*>(raw + (((2u * q + 1u) ^ sw_xor) << 4));
                if (i == 1u) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive(raw_empty(pr.s));
                }
                uint4 o[8];
                decode_row64(c0, c1, i ? sc.y : sc.x, g, o);
                if (i == 0u && u >= u0 + FEW_W_SLOTS) {
                    if (early_w && u < u0 + 2u * FEW_W_SLOTS) grid_dependency_wait();      // first wait for a slot: join the stream's order
                    if (!__all_sync(0xFFFFFFFFu, mbar_wait(w_empty(set), turn ^ 1u, abort_flag))) {
                        atomicOr(a.status, ST_WAIT_EMPTY_DEQ);
                        *abort_flag = 1;
                        ok = false;
                        break;
                    }
                    tc_fence_after_sync();
                }
                uint32_t v[32];
#pragma unroll
                for (uint32_t c = 0; c < 8; c++) {
                    v[4u * c + 0u] = o[c].x;
                    v[4u * c + 1u] = o[c].y;
                    v[4u * c + 2u] = o[c].z;
                    v[4u * c + 3u] = o[c].w;
                }
                tmem_st_32x32b_x32(dst + 32u * i, v);
            }
            if (!ok) break;
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(w_full(set));
        }
        __syncwarp();
        if (early_w) grid_dependency_wait();                                 // r and y belong to the stream's order
    } else if (warp < FEW_WARP_EPI + 4u) {
        // ---------------------------------------------------------------- epilogue of the segments
        const uint32_t row = 32u * (warp & 3u) + lane;
        const uint32_t lane_base = tmem_base + ((32u * (warp & 3u)) << 16);
        uint32_t kb = kb0, tile = tile0;
        for (uint32_t u = u0, seg = 0; u < u1; seg++) {
            const uint32_t set = seg & 1u, len = min(U - kb, u1 - u);
            const bool whole = len == U;
            const uint32_t n_acc = min(ACCS, len * STEPS);
            // (a segment that begins its tile but does not end it is its share's last: the rings are idle by then)
            float* const part = reinterpret_cast<float*>(smem + (kb ? head - base : 0u));
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(acc_full(set), (seg >> 1) & 1u, abort_flag))) {
                atomicOr(a.status, ST_WAIT_ACC);
                *abort_flag = 1;
                break;
            }
            tc_fence_after_sync();
            const size_t col = (size_t)(t_lo + tile) * FEW_ROWS + row;
            for (uint32_t t0 = 0; t0 < a.m; t0 += 8u) {
                float res[8];
                if (whole && a.r) {
#pragma unroll
                    for (uint32_t j = 0; j < 8; j++) res[j] = t0 + j < a.m ? __ldg(a.r + (size_t)(t0 + j) * a.n + col) : 0.0f;
                }
                float s[8];
                constexpr uint32_t AHEAD = ACCS < 4u ? ACCS : 4u;            // accumulators read together (registers)
#pragma unroll
                for (uint32_t a0 = 0; a0 < ACCS; a0 += AHEAD) {
                    if (a0 >= n_acc) break;
                    uint32_t v[AHEAD][8];
#pragma unroll
                    for (uint32_t i = 0; i < AHEAD; i++) tmem_ld_32x32b_x8(lane_base + set * FEW_ACC_SET + (a0 + i) * N + t0, v[i]);
                    tmem_ld_wait();
#pragma unroll
                    for (uint32_t i = 0; i < AHEAD; i++)
#pragma unroll
                        for (uint32_t j = 0; j < 8; j++) s[j] = a0 + i ? s[j] + __uint_as_float(v[i][j]) : __uint_as_float(v[i][j]);
                }
                if (!whole) {
#pragma unroll
                    for (uint32_t j = 0; j < 8; j++)
                        if (t0 + j < a.m) part[(t0 + j) * FEW_ROWS + row] = s[j];
                } else if (a.act != nullptr) {
                    // adjacent lanes hold gate and up of one output: the gate lane finishes the even tokens, the up lane the odd
                    const bool is_up = (lane & 1u) != 0u;
#pragma unroll
                    for (uint32_t j = 0; j < 8; j += 2) {
                        const float recv = __shfl_xor_sync(0xFFFFFFFFu, is_up ? s[j] : s[j + 1u], 1);
                        const float gate = is_up ? recv : s[j], up = is_up ? s[j + 1u] : recv;
                        const uint32_t t = t0 + j + (lane & 1u);
                        if (t < a.m) a.act[(size_t)t * (a.n >> 1) + (col >> 1)] = f32_to_f16_bits(silu_mul_f32(gate, up));
                    }
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 8; j++)
                        if (t0 + j < a.m) a.y[(size_t)(t0 + j) * a.n + col] = a.r ? s[j] + res[j] : s[j];
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(set));
            u += len;
            kb += len;
            if (kb == U) {
                kb = 0;
                tile++;
            }
        }
        __syncwarp();
    }

    tc_fence_before_sync();
    __syncthreads();
    if (C > 1u) {
        cluster_sync_all();                                                  // every block's sums are in its shared memory
        if (warp < FEW_DEQ_WARPS) {
            // the tiles this block has a part of, but not the whole: its first, and its last if that is another
            const uint32_t tile1 = (u1 - 1u) / U, kb1 = u1 - tile1 * U;      // (kb1: 1 .. U)
            for (uint32_t tile = tile0; tile <= tile1; tile++) {
                const bool cut = (tile == tile0 && kb0 != 0u) || (tile == tile1 && kb1 != U);
                if (!cut) continue;
                uint32_t first = 0, last = C - 1u;                           // the blocks that have a part of it
                while (share(first + 1u) <= tile * U) first++;
                while (share(last) >= (tile + 1u) * U) last--;
                const uint32_t P = last - first + 1u;
                const size_t col0 = (size_t)(t_lo + tile) * FEW_ROWS;
                for (uint32_t i = (rank - first) * 512u + tid; i < a.m * 32u; i += P * 512u) {
                    const uint32_t tok = i >> 5, quad = i & 31u, off = tok * (FEW_ROWS * 4u) + quad * 16u;
                    const size_t o = (size_t)tok * a.n + col0 + quad * 4u;
                    float4 s = ld_shared_cluster_f32x4(map_to_cta(base + off, first));
                    auto add = [&](const float4& v) { s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; };
#pragma unroll
                    for (uint32_t c = 1; c < FEW_MAX_CLUSTER; c++)
                        if (c < P) add(ld_shared_cluster_f32x4(map_to_cta(head + off, first + c)));
                    if (a.r) add(__ldg(reinterpret_cast<const float4*>(a.r + o)));
                    if (a.act != nullptr) {
                        reinterpret_cast<uint32_t*>(a.act)[((size_t)tok * (a.n >> 1) + ((col0 + quad * 4u) >> 1)) >> 1] =
                            (uint32_t)f32_to_f16_bits(silu_mul_f32(s.x, s.y)) | ((uint32_t)f32_to_f16_bits(silu_mul_f32(s.z, s.w)) << 16);
                    } else {
                        *reinterpret_cast<float4*>(a.y + o) = s;
                    }
                }
            }
        }
        cluster_sync_all();                                                  // a block's shared memory is read by the others until here
    }
    if (warp == FEW_WARP_MMA) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, PAIR_TMEM_COLS);
    }
}

}  // namespace lexb
