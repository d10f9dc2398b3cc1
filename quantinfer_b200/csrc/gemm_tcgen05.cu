// bfloat16 matrix product on the 5th-generation tensor cores:
//     y[M, N] = x[M, K] . w[N, K]^T        (32-bit accumulation)
// Both operands are read along K ("K-major"), which is the checkpoint's
// [out, in] layout for w, so nothing is transposed at load.
//
// The output is cut into 128 x BN tiles of  D = A . B^T  where A and B are the two
// row-major operands; a CTA computes its share of the tiles one after the other. For many tokens A = x and B = w. For few tokens (decode)
// the operands are swapped: A = w, so the 128 rows of the MMA ride the weight's
// output dimension and the small token count rides the MMA's N (16..256); the
// epilogue then stores the tile transposed. A skinny product is bound by the
// weight stream from HBM, so the K dimension can be split over blockIdx.z to
// put enough CTAs in flight; partial sums go to a 32-bit workspace
// [splits, M, N] and are added in split order by a second kernel (or by the
// consumer: add_rmsnorm takes the partials directly).
//
// Roles inside a CTA (192 threads):
//   warp 0     one lane issues TMA loads (cp.async.bulk.tensor, 128-byte swizzle)
//              into a ring of STAGES shared-memory buffers, each guarded by a
//              "full" mbarrier (expect-tx) and an "empty" mbarrier
//   warp 1     allocates tensor memory; one lane issues tcgen05.mma (kind::f16,
//              M = 128, N = BN, K = 16 per instruction, 4 per 64-wide k block) and
//              tcgen05.commit, which frees the stage and finally signals the
//              accumulator
//   warps 2-5  read the accumulator from tensor memory (tcgen05.ld, 32 lanes x
//              32 columns per warp) and store it
// No load uses cluster multicast. Every mbarrier wait is bounded in time: when
// one runs out the thread sets kStatusWaitTimeout in the status word and an abort
// flag in shared memory, all roles leave their loops and meet, the block waits a
// while for what it still has in flight, tensor memory is freed and the kernel
// returns. A launch that finds the bit set leaves at its first wait that is not
// fulfilled at once. (tcgen05.alloc and the barriers of a block or a cluster have
// no bound of their own: the first waits only for blocks that end, the others
// for roles whose waits do.)
//
// K must be a multiple of 8 (TMA wants row strides of whole 16 bytes); rows of
// A, B and K beyond the tensors are zero-filled by TMA and masked at the store.
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int kThreads = 192;
template <typename TOut> __device__ __forceinline__ void store1(TOut* p, float v);
template <> __device__ __forceinline__ void store1<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void store1<qi::bf16>(qi::bf16* p, float v) { *p = __float2bfloat16_rn(v); }

template <int BN, int STAGES>
struct Smem {
    static constexpr int kABytes = BM * BK * 2;
    static constexpr int kBBytes = BN * BK * 2;
    static constexpr int kStageBytes = kABytes + kBBytes;
    static constexpr int kBarrierBytes = 8 * (2 * STAGES + 4) + 16;
    static constexpr int kTotal = STAGES * kStageBytes + kBarrierBytes + 1024;  // + alignment slack
};


__device__ __forceinline__ float silu_mul(float g, float u) { return g / (1.0f + expf(-g)) * u; }

// What the epilogue of the fused q/k/v projection needs (EPI = 2): the product's columns are
// heads of 128 (nq query heads, then nkv key heads, then nkv value heads); query and key heads
// get their RMSNorm (gain null: none) and the half-split rotation of the token's position (cos_t
// null: none), values pass through; queries go to q_out [tokens, nq * 128], keys and values to
// the token's place in the paged cache (k_pages null: nothing is written).
struct RopeEpilogue {
    qi::bf16* q_out;
    const float* q_gain;
    const float* k_gain;
    const float* cos_t;      // [positions, 64]
    const float* sin_t;
    const int* positions;    // [tokens]
    const int* token_req;    // [tokens]: row of the block table
    const int* block_table;  // [requests, max_blocks]
    qi::bf16* k_pages;       // [pages, nkv, page_size, 128]
    qi::bf16* v_pages;
    float eps;
    int max_blocks, page_size, num_pages, nq, nkv;
    int table_positions;     // rows of cos_t / sin_t
    float limit, alpha;      // EPI = 3 (nothing else of this struct is used there)
};

// The activation of a (gate, up) pair: EPI 1 silu(g) u; EPI 3 the clamped form g sigmoid(alpha g) (u + 1) with g = min(gate,
// limit), u = clamp(up, -limit, limit).
template <int EPI>
__device__ __forceinline__ float pair_act(float g, float u, const RopeEpilogue& e) {
    if (EPI == 1) return silu_mul(g, u);
    g = fminf(g, e.limit);
    u = fminf(fmaxf(u, -e.limit), e.limit);
    return g / (1.0f + expf(-e.alpha * g)) * (u + 1.0f);
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}

// One accumulator tile [128 tokens, BN columns] of the q/k/v projection: this thread owns token
// `row` (TMEM lane) and walks the tile's heads. The norm's sum runs over the head's 128 columns
// in column order; everything is 32-bit until the store.
template <int BN>
__device__ __forceinline__ void rope_epilogue(uint32_t tmem_tile, int col_base, int row, bool row_ok, int n_cols,
                                              const RopeEpilogue& e, int* __restrict__ status) {
    constexpr int D = 128, HALF = 64;
    int pos = row_ok ? e.positions[row] : 0;
    if (pos < 0) {           // no such position: nothing of this token is written
        if (status) atomicOr(status, qi::kStatusBadRange);
        pos = 0;
        row_ok = false;
    }
    int table_row = pos;     // a position beyond the rotation table is flagged and takes the table's last row
    if (e.cos_t && pos >= e.table_positions) {
        if (status) atomicOr(status, qi::kStatusBadRange);
        table_row = e.table_positions - 1;
    }
    int page = -2;           // -2: not looked up yet
#pragma unroll 1
    for (int hh = 0; hh < BN / D; ++hh) {
        const int col0 = col_base + hh * D;
        if (col0 >= n_cols) break;                       // the same for every thread of the CTA
        const int head = col0 / D;
        const bool is_q = head < e.nq, is_k = !is_q && head < e.nq + e.nkv;
        const uint32_t t0 = tmem_tile + (uint32_t)(hh * D);
        const float* gain = is_q ? e.q_gain : is_k ? e.k_gain : nullptr;
        uint32_t lo[32], hi[32];
        float inv = 1.f;
        if (gain) {
            float ss = 0.f;
#pragma unroll 1
            for (int c = 0; c < 4; ++c) {
                tmem_ld32(t0 + 32u * c, lo);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) ss = fmaf(__uint_as_float(lo[i]), __uint_as_float(lo[i]), ss);
            }
            inv = 1.0f / sqrtf(ss / (float)D + e.eps);
        }
        qi::bf16* dst = nullptr;
        if (row_ok) {
            if (is_q) {
                dst = e.q_out + ((size_t)row * e.nq + head) * D;
            } else if (e.k_pages) {
                if (page == -2) {
                    page = e.block_table[(size_t)e.token_req[row] * e.max_blocks + pos / e.page_size];
                    if (page < 0 || page >= e.num_pages) {
                        if (status) atomicOr(status, qi::kStatusBadPage);
                        page = -1;
                    }
                }
                if (page >= 0) {
                    const int hk = is_k ? head - e.nq : head - e.nq - e.nkv;
                    dst = (is_k ? e.k_pages : e.v_pages) + (((size_t)page * e.nkv + hk) * e.page_size + (pos % e.page_size)) * (size_t)D;
                }
            }
        }
        const bool rotate = (is_q || is_k) && e.cos_t != nullptr;
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
            tmem_ld32(t0 + 32u * c, lo);
            tmem_ld32(t0 + (uint32_t)HALF + 32u * c, hi);
            tmem_ld_wait();
            if (!dst) continue;
            float a[32], b[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                a[i] = __uint_as_float(lo[i]);
                b[i] = __uint_as_float(hi[i]);
            }
            if (gain) {
                const float4* ga = reinterpret_cast<const float4*>(gain + 32 * c);
                const float4* gb = reinterpret_cast<const float4*>(gain + HALF + 32 * c);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 x = ga[i], y = gb[i];
                    a[4 * i] = a[4 * i] * inv * x.x; a[4 * i + 1] = a[4 * i + 1] * inv * x.y;
                    a[4 * i + 2] = a[4 * i + 2] * inv * x.z; a[4 * i + 3] = a[4 * i + 3] * inv * x.w;
                    b[4 * i] = b[4 * i] * inv * y.x; b[4 * i + 1] = b[4 * i + 1] * inv * y.y;
                    b[4 * i + 2] = b[4 * i + 2] * inv * y.z; b[4 * i + 3] = b[4 * i + 3] * inv * y.w;
                }
            }
            if (rotate) {
                const float4* cs = reinterpret_cast<const float4*>(e.cos_t + (size_t)table_row * HALF + 32 * c);
                const float4* sn = reinterpret_cast<const float4*>(e.sin_t + (size_t)table_row * HALF + 32 * c);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 cc = cs[i], ss = sn[i];
                    const float cv[4] = {cc.x, cc.y, cc.z, cc.w}, sv[4] = {ss.x, ss.y, ss.z, ss.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float x = a[4 * i + j], y = b[4 * i + j];
                        a[4 * i + j] = x * cv[j] - y * sv[j];
                        b[4 * i + j] = x * sv[j] + y * cv[j];
                    }
                }
            }
            uint4* d_lo = reinterpret_cast<uint4*>(dst + 32 * c);
            uint4* d_hi = reinterpret_cast<uint4*>(dst + HALF + 32 * c);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                d_lo[i] = make_uint4(pack2(a[8 * i], a[8 * i + 1]), pack2(a[8 * i + 2], a[8 * i + 3]),
                                     pack2(a[8 * i + 4], a[8 * i + 5]), pack2(a[8 * i + 6], a[8 * i + 7]));
                d_hi[i] = make_uint4(pack2(b[8 * i], b[8 * i + 1]), pack2(b[8 * i + 2], b[8 * i + 3]),
                                     pack2(b[8 * i + 4], b[8 * i + 5]), pack2(b[8 * i + 6], b[8 * i + 7]));
            }
        }
    }
}

// EPI = 0: store the product. EPI = 1: the product's columns come in pairs (gate, up) and
// the kernel stores silu(gate) * up, half as wide (the feed-forward's activation fused in).
// EPI = 3: the same pairs through the clamped gated form.
// EPI = 2 (operands not swapped): the product is the q/k/v projection and `rope` says where
// its heads go (q/k norm, rotation and the cache write fused in; `out` is not used).
//
// The kernel is persistent: CTA c takes tiles c, c + gridDim.x, ... of the linear tile
// list (A tiles fastest, then B tiles, then K splits, so CTAs that run together share a
// B tile in L2). The accumulator in tensor memory is double-buffered: while the
// epilogue warps drain one buffer, the MMA warp already fills the other with the next
// tile, and the TMA ring runs on across tile borders.
QI_TL_DEFINE(qi_timeline_gemm)

template <int BN, int STAGES, bool SWAP, typename TOut, int EPI>
__global__ void __launch_bounds__(kThreads)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    TOut* __restrict__ out, int rows_a, int rows_b, int K, long long ld_out,
                    int kb_per_split, int n_splits, long long split_stride, int* __restrict__ status,
                    const RopeEpilogue rope) {
    extern __shared__ uint8_t smem_raw[];
    using L = Smem<BN, STAGES>;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    // barriers: full[STAGES], empty[STAGES], acc_full[2], acc_empty[2]
    const uint32_t bars = base + STAGES * L::kStageBytes;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aligned + STAGES * L::kStageBytes + 8 * (2 * STAGES + 4));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
    auto acc_full_bar = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto acc_empty_bar = [&](int a) { return bars + 8u * (2 * STAGES + 2 + a); };

    QI_TL_BEGIN();
    QI_TL_SHARED();
    qi::pdl_launch_dependents();   // the next kernel may be scheduled while this one runs
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles_a = (rows_a + BM - 1) / BM, tiles_b = (rows_b + BN - 1) / BN;
    const int total_tiles = tiles_a * tiles_b * n_splits;
    const int kb_total = (K + BK - 1) / BK;
    constexpr uint32_t kAccCols = BN < 32 ? 32 : BN;        // columns of one accumulator
    constexpr uint32_t kTmemCols = 2 * kAccCols;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full_bar(a), 1);
            mbar_init(acc_empty_bar(a), 4);     // one arrival per epilogue warp
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    // Set-up is done. Only the activations (and the output buffer) depend on the kernel before
    // this one: the producer fetches the first weight tiles before it waits for that kernel, the
    // epilogue warps wait before they write, and the MMA warp follows the producer's barriers.

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            // The weights are the operand with the many rows: A when the operands are swapped
            // (few tokens), else B. They are never written on the device, so the first stages'
            // weight tiles of this CTA's first tile are requested before the wait.
            const uint64_t stream_once = l2_evict_first_policy();
            uint32_t early = 0;
            if (blockIdx.x < total_tiles) {
                const int tile = blockIdx.x;
                const int tile_a = tile % tiles_a, tile_b = (tile / tiles_a) % tiles_b, split = tile / (tiles_a * tiles_b);
                const int kb_begin = split * kb_per_split;
                const int n_kb = max(min(kb_total, kb_begin + kb_per_split) - kb_begin, 0);
                early = (uint32_t)min(n_kb, STAGES);
                for (uint32_t i = 0; i < early; ++i) {
                    mbar_expect_tx(full_bar(i), L::kStageBytes);
                    const uint32_t a_dst = base + i * L::kStageBytes;
                    const int k0 = (kb_begin + (int)i) * BK;
                    if (SWAP) tma_load_2d_hint(a_dst, &map_a, full_bar(i), k0, tile_a * BM, stream_once);
                    else tma_load_2d(a_dst + L::kABytes, &map_b, full_bar(i), k0, tile_b * BN);
                }
            }
            qi::pdl_wait();
            uint32_t it = 0;          // k blocks issued so far, over all tiles
            bool ok = true;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x) {
                const int tile_a = tile % tiles_a, tile_b = (tile / tiles_a) % tiles_b, split = tile / (tiles_a * tiles_b);
                const int kb_begin = split * kb_per_split;
                const int n_kb = max(min(kb_total, kb_begin + kb_per_split) - kb_begin, 0);
                for (int i = 0; i < n_kb; ++i, ++it) {
                    const int s = it % STAGES;
                    const uint32_t a_dst = base + s * L::kStageBytes;
                    const int k0 = (kb_begin + i) * BK;
                    if (it < early) {
                        // the weight tile of this stage is on its way already: add the activations
                        if (SWAP) tma_load_2d(a_dst + L::kABytes, &map_b, full_bar(s), k0, tile_b * BN);
                        else tma_load_2d(a_dst, &map_a, full_bar(s), k0, tile_a * BM);
                        continue;
                    }
                    if (!mbar_wait(empty_bar(s), ((it / STAGES) & 1u) ^ 1u, abort_flag, status)) {
                        give_up(abort_flag, status);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(full_bar(s), L::kStageBytes);
                    if (SWAP) tma_load_2d_hint(a_dst, &map_a, full_bar(s), k0, tile_a * BM, stream_once);
                    else tma_load_2d(a_dst, &map_a, full_bar(s), k0, tile_a * BM);
                    tma_load_2d(a_dst + L::kABytes, &map_b, full_bar(s), k0, tile_b * BN);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            qi::pdl_wait();   // its operands come after the producer's wait: the polls below start counting from there
            QI_TL_SHARED_WAKE();
            constexpr uint32_t idesc = make_idesc(BM, BN);
            uint32_t it = 0;
            int j = 0;                // tiles this CTA has started
            bool ok = true;
            for (int tile = blockIdx.x; tile < total_tiles && ok; tile += gridDim.x, ++j) {
                const int split = tile / (tiles_a * tiles_b);
                const int kb_begin = split * kb_per_split;
                const int n_kb = max(min(kb_total, kb_begin + kb_per_split) - kb_begin, 0);
                const int acc = j & 1;
                // the epilogue must have drained this accumulator (first use of each passes at once)
                if (!mbar_wait(acc_empty_bar(acc), (((uint32_t)j >> 1) & 1u) ^ 1u, abort_flag, status)) {
                    give_up(abort_flag, status);
                    break;
                }
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + (uint32_t)acc * kAccCols;
                for (int i = 0; i < n_kb; ++i, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(full_bar(s), (it / STAGES) & 1u, abort_flag, status)) {
                        give_up(abort_flag, status);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    if (it == 0) QI_TL_SHARED_DATA();
                    const uint32_t a_addr = base + s * L::kStageBytes;
                    const uint64_t adesc = make_smem_desc(a_addr);
                    const uint64_t bdesc = make_smem_desc(a_addr + L::kABytes);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) {
                        // 16 bf16 = 32 bytes further along the swizzled row: +2 in units of 16 bytes
                        umma_bf16(tmem_d, adesc + 2u * k, bdesc + 2u * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit(empty_bar(s));   // the stage is free once these MMAs have read it
                }
                if (ok) umma_commit(acc_full_bar(acc));  // the accumulator is complete
            }
        }
    } else {
        // ---------------- epilogue (warps 2..5) ----------------
        const int quarter = warp & 3;   // the 32 TMEM lanes this warp may read
        qi::pdl_wait();                 // the output buffer may still be read by the kernel before
        if (threadIdx.x == 64 && failed_before(status)) give_up(abort_flag, status);
        int j = 0;
        for (int tile = blockIdx.x; tile < total_tiles; tile += gridDim.x, ++j) {
            const int tile_a = tile % tiles_a, tile_b = (tile / tiles_a) % tiles_b, split = tile / (tiles_a * tiles_b);
            const int kb_begin = split * kb_per_split;
            const int n_kb = max(min(kb_total, kb_begin + kb_per_split) - kb_begin, 0);
            const int acc = j & 1;
            if (!mbar_wait_warp(acc_full_bar(acc), ((uint32_t)j >> 1) & 1u, abort_flag, status)) {
                if (lane == 0) give_up(abort_flag, status);
                break;
            }
            tc_fence_after();
            const int a_row = tile_a * BM + quarter * 32 + lane;
            if constexpr (EPI == 2 && BN % 128 == 0) {
                rope_epilogue<BN>(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)acc * kAccCols, tile_b * BN, a_row,
                                  a_row < rows_a, rows_b, rope, status);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty_bar(acc));
                continue;
            }
            TOut* obase = out + (size_t)split * split_stride;
            constexpr int kChunk = BN >= 32 ? 32 : 16;
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += kChunk) {
                uint32_t r[32];
                if (n_kb > 0) {
                    const uint32_t addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)acc * kAccCols + (uint32_t)c0;
                    if (kChunk == 32) tmem_ld32(addr, r); else tmem_ld16(addr, r);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int q = 0; q < 32; ++q) r[q] = 0u;   // an empty K range contributes zeros
                }
                if (c0 + kChunk >= BN) {
                    // everything of this accumulator is in registers: hand it back to the MMA warp
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_empty_bar(acc));
                }
                const int b0 = tile_b * BN + c0;
                if (b0 >= rows_b) continue;       // (the same for every thread: a chunk of no tokens)
                if (SWAP && (EPI == 1 || EPI == 3)) {
                    // Rows of A come in pairs (gate, up), one a lane. Of two columns a lane keeps one and gives the other to its
                    // neighbour: even lanes compute column q, odd lanes q + 1. All values are computed before any is
                    // stored: with a branch around each, nothing hid the exponential and the division (36 layers of
                    // [33, 4096] . [24576, 4096]^T in their step: 3,951 -> 3,859 us, with 64 tokens 5,044 -> 4,819 us).
                    const bool odd = lane & 1;
                    float v[kChunk / 2];
#pragma unroll
                    for (int q = 0; q < kChunk / 2; ++q) {
                        const float keep = __uint_as_float(odd ? r[2 * q + 1] : r[2 * q]);
                        const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(odd ? r[2 * q] : r[2 * q + 1]), 1);
                        v[q] = pair_act<EPI>(odd ? got : keep, odd ? keep : got, rope);
                    }
                    const int b = b0 + (odd ? 1 : 0);
                    if ((a_row | 1) < rows_a) {
                        TOut* o = obase + (size_t)b * ld_out + (a_row >> 1);
#pragma unroll
                        for (int q = 0; q < kChunk / 2; ++q) {
                            if (b + 2 * q < rows_b) store1<TOut>(o, v[q]);
                            o += 2 * ld_out;
                        }
                    }
                    __syncwarp();
                } else if (SWAP) {
                    // out[b, a]: for a fixed column the warp's lanes write consecutive addresses
                    if (a_row < rows_a) {
#pragma unroll
                        for (int q = 0; q < kChunk; ++q)
                            if (b0 + q < rows_b) store1<TOut>(obase + (size_t)(b0 + q) * ld_out + a_row, __uint_as_float(r[q]));
                    }
                } else if (EPI == 1 || EPI == 3) {
                    if (a_row < rows_a) {
                        TOut* orow = obase + (size_t)a_row * ld_out + (b0 >> 1);
                        const bool full = b0 + kChunk <= rows_b;
                        const bool aligned16 = ((reinterpret_cast<uintptr_t>(orow) & 15u) == 0);
                        if (full && aligned16 && sizeof(TOut) == 2) {
#pragma unroll
                            for (int q0 = 0; q0 < kChunk; q0 += 16) {
                                uint4 v;
                                uint32_t* vw = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
                                for (int q = 0; q < 4; ++q) {
                                    __nv_bfloat162 pr = __floats2bfloat162_rn(
                                        pair_act<EPI>(__uint_as_float(r[q0 + 4 * q]), __uint_as_float(r[q0 + 4 * q + 1]), rope),
                                        pair_act<EPI>(__uint_as_float(r[q0 + 4 * q + 2]), __uint_as_float(r[q0 + 4 * q + 3]), rope));
                                    vw[q] = *reinterpret_cast<uint32_t*>(&pr);
                                }
                                *reinterpret_cast<uint4*>(reinterpret_cast<qi::bf16*>(orow) + (q0 >> 1)) = v;
                            }
                        } else {
#pragma unroll
                            for (int q = 0; q < kChunk; q += 2)
                                if (b0 + q + 1 < rows_b)
                                    store1<TOut>(orow + (q >> 1), pair_act<EPI>(__uint_as_float(r[q]), __uint_as_float(r[q + 1]), rope));
                        }
                    }
                } else {
                    if (a_row < rows_a) {
                        TOut* orow = obase + (size_t)a_row * ld_out + b0;
                        const bool full = b0 + kChunk <= rows_b;
                        const bool aligned16 = ((reinterpret_cast<uintptr_t>(orow) & 15u) == 0);
                        if (full && aligned16 && sizeof(TOut) == 2) {
#pragma unroll
                            for (int q = 0; q < kChunk; q += 8) {
                                uint4 v;
                                __nv_bfloat162 p0 = __floats2bfloat162_rn(__uint_as_float(r[q + 0]), __uint_as_float(r[q + 1]));
                                __nv_bfloat162 p1 = __floats2bfloat162_rn(__uint_as_float(r[q + 2]), __uint_as_float(r[q + 3]));
                                __nv_bfloat162 p2 = __floats2bfloat162_rn(__uint_as_float(r[q + 4]), __uint_as_float(r[q + 5]));
                                __nv_bfloat162 p3 = __floats2bfloat162_rn(__uint_as_float(r[q + 6]), __uint_as_float(r[q + 7]));
                                v.x = *reinterpret_cast<uint32_t*>(&p0);
                                v.y = *reinterpret_cast<uint32_t*>(&p1);
                                v.z = *reinterpret_cast<uint32_t*>(&p2);
                                v.w = *reinterpret_cast<uint32_t*>(&p3);
                                *reinterpret_cast<uint4*>(reinterpret_cast<qi::bf16*>(orow) + q) = v;
                            }
                        } else if (full && aligned16 && sizeof(TOut) == 4) {
#pragma unroll
                            for (int q = 0; q < kChunk; q += 4) {
                                uint4 v = make_uint4(r[q], r[q + 1], r[q + 2], r[q + 3]);
                                *reinterpret_cast<uint4*>(reinterpret_cast<float*>(orow) + q) = v;
                            }
                        } else {
#pragma unroll
                            for (int q = 0; q < kChunk; ++q)
                                if (b0 + q < rows_b) store1<TOut>(orow + q, __uint_as_float(r[q]));
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1 && *abort_flag) settle_in_flight();
    QI_TL_END_SHARED(20 + EPI + (SWAP ? 0 : 5));
    if (warp == 1) tmem_dealloc(tmem_base, kTmemCols);
}

// ------------------------------------------------------------------ two CTAs on one tile
//
// For many tokens the single-CTA kernel is bound by what its 128 x 256 tiles draw from L2 and
// shared memory (48 KB per 64-wide k block for 512 cycles of tensor-core work) rather than
// by the tensor core. Here a pair of CTAs on neighbouring SMs (a cluster of two) computes one
// 256 x 256 tile with tcgen05.mma.cta_group::2: each CTA loads 128 rows of A and 128 rows of
// B (32 KB per k block, six stages instead of four), the tensor cores of both SMs read B
// from both CTAs' shared memory, and each CTA's tensor memory receives its 128 rows of the
// result. Only the even CTA of the pair issues MMAs. Barriers:
//   full[s]   in the even CTA: its producer announces the bytes of both CTAs' copies, and
//             both CTAs' TMA copies report there (cta_group::2 form of the copy)
//   empty[s]  in each CTA: the MMAs' commit arrives on both (multicast commit, not a load)
//   acc_full  in each CTA: the same at the end of a tile
//   acc_empty in the even CTA: the four epilogue warps of both CTAs arrive there
// No load uses cluster multicast. All waits are bounded as in the kernel above; a CTA that
// gives up says so in its partner's shared memory too. Both CTAs pass a cluster barrier
// before they leave, so that neither frees shared or tensor memory its partner still uses.

constexpr int kPairStages = 6;
constexpr int kPairHalfBytes = BM * BK * 2;              // 128 rows x 64 bf16 = 16 KB
constexpr int kPairStageBytes = 2 * kPairHalfBytes;      // this CTA's rows of A, then its rows of B
constexpr int kPairSmem = kPairStages * kPairStageBytes + 8 * (2 * kPairStages + 4) + 16 + 1024;

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {      // (not .aligned: a role's one lane comes after the rest of its warp)
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The copy of a CTA of a pair; its bytes are reported to the barrier at the same address in the even CTA.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar & 0xFEFFFFFFu), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t dst_smem, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t addr, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8, %9, %10, %11, %12}, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0), "r"(0), "r"(0), "r"(0), "r"(0), "r"(0),
          "r"(0), "r"(0) : "memory");
}
// Arrives on the barrier at this address in both CTAs of the pair when every MMA issued so far has completed.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
}
// Arrives on the barrier at this address in the even CTA of the pair.
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .b32 ra;\n\t"
        "mapa.shared::cluster.u32 ra, %0, 0;\n\t"
        "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [ra];\n\t}"
        ::"r"(bar) : "memory");
}

// As give_up(), in both CTAs of the pair: each reads the other's shared memory until the last MMA has run.
__device__ __forceinline__ void give_up_pair(volatile int* abort_flag, int* status, uint32_t rank) {
    if (*abort_flag) return;
    give_up(abort_flag, status);
    asm volatile(
        "{\n\t.reg .b32 ra;\n\t"
        "mapa.shared::cluster.u32 ra, %0, %1;\n\t"
        "st.shared::cluster.u32 [ra], %2;\n\t}"
        ::"r"(smem_u32(const_cast<const int*>(abort_flag))), "r"(rank ^ 1u), "r"(1) : "memory");
}

// out[M, N] = A[M, K] . B[N, K]^T in tiles of 256 x 256, one per pair of CTAs at a time; A are the
// tokens, B the weights. EPI as in the kernel above (0: the product, 1: silu(gate) * up of column
// pairs, 2: the q/k/v projection's heads through `rope`, 3: the clamped form of the pairs).
template <typename TOut, int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads)
gemm_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                         TOut* __restrict__ out, int rows_a, int rows_b, int K, long long ld_out, int kb_per_split,
                         int n_splits, long long split_stride, int* __restrict__ status, const RopeEpilogue rope) {
    extern __shared__ uint8_t smem_raw[];
    constexpr int STAGES = kPairStages;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + STAGES * kPairStageBytes;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aligned + STAGES * kPairStageBytes + 8 * (2 * STAGES + 4));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
    auto acc_full_bar = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto acc_empty_bar = [&](int a) { return bars + 8u * (2 * STAGES + 2 + a); };

    QI_TL_BEGIN();
    qi::pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    constexpr int TM = 2 * BM, TN = 256;
    const int tiles_m = (rows_a + TM - 1) / TM, tiles_n = (rows_b + TN - 1) / TN;
    const int total_tiles = tiles_m * tiles_n * n_splits;     // K splits slowest: split s writes out + s * split_stride
    const int kb_total = (K + BK - 1) / BK;
    auto kb_range = [&](int tile, int& kb_begin) {
        kb_begin = (tile / (tiles_m * tiles_n)) * kb_per_split;
        return max(min(kb_total, kb_begin + kb_per_split) - kb_begin, 0);
    };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full_bar(a), 1);
            mbar_init(acc_empty_bar(a), 8);     // four epilogue warps in each CTA of the pair
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(tmem_slot), 512);
        tmem_relinquish_pair();
    }
    tc_fence_before();
    cluster_sync_all();       // both CTAs' barriers and tensor memory exist before anything crosses over
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer (in both CTAs) ----------------
        if (lane == 0) {
            // the first stages' weight rows are requested before the wait for the kernel before this one
            uint32_t early = 0;
            if (pair < total_tiles) {
                const int tile_n = (pair / tiles_m) % tiles_n;
                int kb_begin;
                const int n_kb = kb_range(pair, kb_begin);
                early = (uint32_t)min(n_kb, STAGES);
                for (uint32_t i = 0; i < early; ++i) {
                    if (rank == 0) mbar_expect_tx(full_bar(i), 2 * kPairStageBytes);
                    tma_load_2d_pair(base + i * kPairStageBytes + kPairHalfBytes, &map_b, full_bar(i), (kb_begin + (int)i) * BK,
                                     tile_n * TN + (int)rank * BM);
                }
            }
            qi::pdl_wait();
            QI_TL_WAKE();
            uint32_t it = 0;
            bool ok = true;
            for (int tile = pair; tile < total_tiles && ok; tile += n_pairs) {
                const int tile_m = tile % tiles_m, tile_n = (tile / tiles_m) % tiles_n;
                int kb_begin;
                const int n_kb = kb_range(tile, kb_begin);
                for (int i = 0; i < n_kb; ++i, ++it) {
                    const int s = it % STAGES;
                    const uint32_t dst = base + s * kPairStageBytes;
                    const int k0 = (kb_begin + i) * BK;
                    if (it < early) {
                        tma_load_2d_pair(dst, &map_a, full_bar(s), k0, tile_m * TM + (int)rank * BM);
                        continue;
                    }
                    if (!mbar_wait(empty_bar(s), ((it / STAGES) & 1u) ^ 1u, abort_flag, status)) {
                        give_up_pair(abort_flag, status, rank);
                        ok = false;
                        break;
                    }
                    if (rank == 0) mbar_expect_tx(full_bar(s), 2 * kPairStageBytes);
                    tma_load_2d_pair(dst, &map_a, full_bar(s), k0, tile_m * TM + (int)rank * BM);
                    tma_load_2d_pair(dst + kPairHalfBytes, &map_b, full_bar(s), k0, tile_n * TN + (int)rank * BM);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (the even CTA only) ----------------
        if (lane == 0 && rank == 0) {
            qi::pdl_wait();
            constexpr uint32_t idesc = make_idesc(TM, TN);
            uint32_t it = 0;
            int j = 0;
            bool ok = true;
            for (int tile = pair; tile < total_tiles && ok; tile += n_pairs, ++j) {
                const int acc = j & 1;
                int kb_begin;
                const int n_kb = kb_range(tile, kb_begin);
                if (!mbar_wait(acc_empty_bar(acc), (((uint32_t)j >> 1) & 1u) ^ 1u, abort_flag, status)) {
                    give_up_pair(abort_flag, status, rank);
                    break;
                }
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + (uint32_t)acc * TN;
                for (int i = 0; i < n_kb; ++i, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(full_bar(s), (it / STAGES) & 1u, abort_flag, status)) {
                        give_up_pair(abort_flag, status, rank);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_addr = base + s * kPairStageBytes;
                    const uint64_t adesc = make_smem_desc(a_addr);
                    const uint64_t bdesc = make_smem_desc(a_addr + kPairHalfBytes);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k)
                        umma_bf16_pair(tmem_d, adesc + 2u * k, bdesc + 2u * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
                    umma_commit_pair(empty_bar(s));
                }
                if (ok) umma_commit_pair(acc_full_bar(acc));
            }
        }
    } else {
        // ---------------- epilogue (warps 2..5 of both CTAs): this CTA's 128 rows of the tile ----------------
        const int quarter = warp & 3;
        qi::pdl_wait();
        if (threadIdx.x == 64 && failed_before(status)) give_up_pair(abort_flag, status, rank);
        int j = 0;
        for (int tile = pair; tile < total_tiles; tile += n_pairs, ++j) {
            const int tile_m = tile % tiles_m, tile_n = (tile / tiles_m) % tiles_n;
            TOut* obase = out + (size_t)(tile / (tiles_m * tiles_n)) * split_stride;
            const int acc = j & 1;
            if (!mbar_wait_warp(acc_full_bar(acc), ((uint32_t)j >> 1) & 1u, abort_flag, status)) {
                if (lane == 0) give_up_pair(abort_flag, status, rank);
                break;
            }
            tc_fence_after();
            const int row = tile_m * TM + (int)rank * BM + quarter * 32 + lane;
            const uint32_t tmem_tile = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)acc * TN;
            if constexpr (EPI == 2) {
                rope_epilogue<TN>(tmem_tile, tile_n * TN, row, row < rows_a, rows_b, rope, status);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_leader(acc_empty_bar(acc));
                continue;
            }
#pragma unroll 1
            for (int c0 = 0; c0 < TN; c0 += 32) {
                uint32_t r[32];
                tmem_ld32(tmem_tile + (uint32_t)c0, r);
                tmem_ld_wait();
                if (c0 + 32 >= TN) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_leader(acc_empty_bar(acc));
                }
                const int b0 = tile_n * TN + c0;
                if (row >= rows_a) continue;
                const bool full = b0 + 32 <= rows_b;
                if (EPI == 1 || EPI == 3) {
                    // columns come in pairs (gate, up): half as many outputs
                    TOut* orow = obase + (size_t)row * ld_out + (b0 >> 1);
                    if (full && ((reinterpret_cast<uintptr_t>(orow) & 15u) == 0) && sizeof(TOut) == 2) {
#pragma unroll
                        for (int q0 = 0; q0 < 32; q0 += 16) {
                            uint4 v;
                            v.x = pack2(pair_act<EPI>(__uint_as_float(r[q0 + 0]), __uint_as_float(r[q0 + 1]), rope),
                                        pair_act<EPI>(__uint_as_float(r[q0 + 2]), __uint_as_float(r[q0 + 3]), rope));
                            v.y = pack2(pair_act<EPI>(__uint_as_float(r[q0 + 4]), __uint_as_float(r[q0 + 5]), rope),
                                        pair_act<EPI>(__uint_as_float(r[q0 + 6]), __uint_as_float(r[q0 + 7]), rope));
                            v.z = pack2(pair_act<EPI>(__uint_as_float(r[q0 + 8]), __uint_as_float(r[q0 + 9]), rope),
                                        pair_act<EPI>(__uint_as_float(r[q0 + 10]), __uint_as_float(r[q0 + 11]), rope));
                            v.w = pack2(pair_act<EPI>(__uint_as_float(r[q0 + 12]), __uint_as_float(r[q0 + 13]), rope),
                                        pair_act<EPI>(__uint_as_float(r[q0 + 14]), __uint_as_float(r[q0 + 15]), rope));
                            *reinterpret_cast<uint4*>(reinterpret_cast<qi::bf16*>(orow) + (q0 >> 1)) = v;
                        }
                    } else {
#pragma unroll
                        for (int q = 0; q < 32; q += 2)
                            if (b0 + q + 1 < rows_b)
                                store1<TOut>(orow + (q >> 1), pair_act<EPI>(__uint_as_float(r[q]), __uint_as_float(r[q + 1]), rope));
                    }
                } else {
                    TOut* orow = obase + (size_t)row * ld_out + b0;
                    if (full && ((reinterpret_cast<uintptr_t>(orow) & 15u) == 0) && sizeof(TOut) == 2) {
#pragma unroll
                        for (int q = 0; q < 32; q += 8) {
                            uint4 v;
                            v.x = pack2(__uint_as_float(r[q + 0]), __uint_as_float(r[q + 1]));
                            v.y = pack2(__uint_as_float(r[q + 2]), __uint_as_float(r[q + 3]));
                            v.z = pack2(__uint_as_float(r[q + 4]), __uint_as_float(r[q + 5]));
                            v.w = pack2(__uint_as_float(r[q + 6]), __uint_as_float(r[q + 7]));
                            *reinterpret_cast<uint4*>(reinterpret_cast<qi::bf16*>(orow) + q) = v;
                        }
                    } else if (full && ((reinterpret_cast<uintptr_t>(orow) & 15u) == 0) && sizeof(TOut) == 4) {
#pragma unroll
                        for (int q = 0; q < 32; q += 4)
                            *reinterpret_cast<uint4*>(reinterpret_cast<float*>(orow) + q) = make_uint4(r[q], r[q + 1], r[q + 2], r[q + 3]);
                    } else {
#pragma unroll
                        for (int q = 0; q < 32; ++q)
                            if (b0 + q < rows_b) store1<TOut>(orow + q, __uint_as_float(r[q]));
                    }
                }
            }
        }
    }
    tc_fence_before();
    cluster_sync_all();       // neither CTA goes before its partner is done with what it holds
    if (warp == 1 && *abort_flag) settle_in_flight();
    QI_TL_END(25 + EPI);
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// ------------------------------------------------------------------ weights on the rows of CTA pairs, grouped
//
// The products of a mixture of experts in ONE launch: group e's rows of x [rows, K] (offsets[e] .. offsets[e + 1] - 1,
// read on the device) times its own weights w[e] [N, K]. A pair of CTAs computes 256 weight rows x up to 256 tokens
// with tcgen05.mma.cta_group::2; the tokens ride the MMA's N, whose width is set for every tile: a group's rows
// are cut into ceil(rows / 256) tiles of equal width, rounded up to 32, so that 190 rows cost 192 columns and 530
// cost 3 x 192, where rows of 128 or 256 would cost 256 and 640 or 768. The tile list (groups, then
// weight tiles, then token tiles: pairs that run together share weights in L2) is walked from the offsets, so no count
// crosses to the host and the step may sit in a graph.
// Bound by the L2's rate into the SMs (32 KB of weights and 128 bytes a token a k block and pair: 10 TB/s measured), by the weights' way in
// from HBM below about 100 rows a group. Columns of a tile beyond its rows hold other rows' results and are not stored; weight rows
// beyond N belong to the next group and are not stored either. Eight epilogue warps, two a quarter of tensor memory: with four, the
// activation of a tile took longer than its products at K = 2,048 (139 -> 121 us there).
// Measured against one dense launch an expert over four streams, which this replaced: gate, up and down of 16 experts
// of 2,048 (2,048 hidden, 4 a token, 2,048 tokens) 405 -> 187 us; of 32 experts of 1,536 (4,096 hidden, 1,537 tokens) 420 -> 273 us,
// where the weights alone take 187 us of HBM time.
// Barriers, roles and bounds as in the kernel of pairs above, except that a CTA takes nothing (no tensor memory, no part in a barrier of the
// pair) before the kernel ahead has ended, and lets the next one start only then. A dense form that took these early, and asked for its
// first weights then, hung in a step of 647 tokens through sizes of 4,096 (no wait on an mbarrier ran out; which wait it was is not known).
// The producer's rate of issue counts: a CTA's half of a tile's tokens (16, 32, ... 128 rows) is ONE copy, with a tensor map
// for every height. As copies of 32 rows each, four a k block, the kernel ran at half the rate.
struct WideMaps { CUtensorMap of[8]; };      // of[i]: boxes of 16 (i + 1) tokens
constexpr int kWideMaxGroups = 1024;
constexpr int kWideSmem = kPairSmem + 4 * (kWideMaxGroups + 1) + 12;
constexpr int kWideThreads = 320;            // producer, MMA, eight epilogue warps

struct WideTile { int group, row0, rows, width, n0; };    // tokens row0 .. row0 + rows - 1 on `width` columns, weight rows from n0

// Walks the tile list in ascending order.
struct WideWalk {
    const int* off;
    int groups, tiles_w, n_rows;
    int group = 0, base = 0;        // the group reached and the tiles before it
    __device__ __forceinline__ bool locate(int tile, WideTile& t) {
        for (; group < groups; ++group) {
            const int first = min(max(off[group], 0), n_rows);
            const int rows = min(max(off[group + 1], first), n_rows) - first;
            const int parts = (rows + 255) >> 8, n = parts * tiles_w;
            if (tile < base + n) {
                const int at = tile - base, part = at % parts;
                const int width = ((rows + parts - 1) / parts + 31) & ~31;
                t.group = group;
                t.row0 = first + part * width;
                t.rows = min(width, rows - part * width);
                t.width = (max(t.rows, 1) + 31) & ~31;
                t.n0 = (at / parts) * (2 * BM);
                return true;
            }
            base += n;
        }
        return false;
    }
};

template <int EPI>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kWideThreads)
gemm_tcgen05_grouped_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ WideMaps maps_x,
                            qi::bf16* __restrict__ out, const int* __restrict__ offsets, int groups, int n_rows, int N, int K,
                            long long ld_out, int* __restrict__ status, const RopeEpilogue act) {
    extern __shared__ uint8_t smem_raw[];
    constexpr int STAGES = kPairStages;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + STAGES * kPairStageBytes;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aligned + STAGES * kPairStageBytes + 8 * (2 * STAGES + 4));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* off = reinterpret_cast<int*>(tmem_slot + 4);
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (STAGES + s); };
    auto acc_full_bar = [&](int a) { return bars + 8u * (2 * STAGES + a); };
    auto acc_empty_bar = [&](int a) { return bars + 8u * (2 * STAGES + 2 + a); };

    QI_TL_BEGIN();
    qi::pdl_wait();
    qi::pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int pair = blockIdx.x >> 1, n_pairs = gridDim.x >> 1;
    const int n_kb = (K + BK - 1) / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full_bar(a), 1);
            mbar_init(acc_empty_bar(a), 16);    // eight epilogue warps in each CTA of the pair
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc_pair(smem_u32(tmem_slot), 512);
        tmem_relinquish_pair();
    }
    for (int i = threadIdx.x; i <= groups; i += kWideThreads) off[i] = offsets[i];
    tc_fence_before();
    cluster_sync_all();       // both CTAs' barriers and tensor memory exist before anything crosses over
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    WideWalk walk{off, groups, (N + 2 * BM - 1) / (2 * BM), n_rows};
    WideTile t;

    if (warp == 0) {
        // ---------------- TMA producer (in both CTAs) ----------------
        if (lane == 0) {
            uint32_t it = 0;
            bool ok = true;
            for (int tile = pair; ok && walk.locate(tile, t); tile += n_pairs) {
                const int half = t.width >> 1;
                const CUtensorMap* map_x = &maps_x.of[(half >> 4) - 1];
                const uint32_t bytes = 2u * (kPairHalfBytes + (uint32_t)half * BK * 2);
                const int w_row = t.group * N + t.n0 + (int)rank * BM, x_row = t.row0 + (int)rank * half;
                for (int i = 0; i < n_kb; ++i, ++it) {
                    const int s = it % STAGES;
                    const uint32_t dst = base + s * kPairStageBytes;
                    if (!mbar_wait(empty_bar(s), ((it / STAGES) & 1u) ^ 1u, abort_flag, status)) {
                        give_up_pair(abort_flag, status, rank);
                        ok = false;
                        break;
                    }
                    if (rank == 0) mbar_expect_tx(full_bar(s), bytes);
                    tma_load_2d_pair(dst, &map_w, full_bar(s), i * BK, w_row);
                    tma_load_2d_pair(dst + kPairHalfBytes, map_x, full_bar(s), i * BK, x_row);
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (the even CTA only) ----------------
        if (lane == 0 && rank == 0) {
            uint32_t it = 0;
            int j = 0;
            bool ok = true;
            for (int tile = pair; ok && walk.locate(tile, t); tile += n_pairs, ++j) {
                const int acc = j & 1;
                const uint32_t idesc = make_idesc(2 * BM, t.width);
                if (!mbar_wait(acc_empty_bar(acc), (((uint32_t)j >> 1) & 1u) ^ 1u, abort_flag, status)) {
                    give_up_pair(abort_flag, status, rank);
                    break;
                }
                tc_fence_after();
                const uint32_t tmem_d = tmem_base + (uint32_t)acc * 256u;
                for (int i = 0; i < n_kb; ++i, ++it) {
                    const int s = it % STAGES;
                    if (!mbar_wait(full_bar(s), (it / STAGES) & 1u, abort_flag, status)) {
                        give_up_pair(abort_flag, status, rank);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a_addr = base + s * kPairStageBytes;
                    const uint64_t adesc = make_smem_desc(a_addr);
                    const uint64_t bdesc = make_smem_desc(a_addr + kPairHalfBytes);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k)
                        umma_bf16_pair(tmem_d, adesc + 2u * k, bdesc + 2u * k, idesc, (i > 0 || k > 0) ? 1u : 0u);
                    umma_commit_pair(empty_bar(s));
                }
                if (ok) umma_commit_pair(acc_full_bar(acc));
            }
        }
    } else {
        // ---------------- epilogue (warps 2..9 of both CTAs): this CTA's 128 weight rows of the tile ----------------
        const int quarter = warp & 3, set = (warp - 2) >> 2;       // a quarter's two warps take chunks of 32 columns in turn
        const bool odd = lane & 1;
        if (threadIdx.x == 64 && failed_before(status)) give_up_pair(abort_flag, status, rank);
        int j = 0;
        for (int tile = pair; walk.locate(tile, t); tile += n_pairs, ++j) {
            const int acc = j & 1;
            if (!mbar_wait_warp(acc_full_bar(acc), ((uint32_t)j >> 1) & 1u, abort_flag, status)) {
                if (lane == 0) give_up_pair(abort_flag, status, rank);
                break;
            }
            tc_fence_after();
            const int n = t.n0 + (int)rank * BM + quarter * 32 + (lane & ~1);      // a lane and its neighbour hold weight rows n, n + 1 (N is even)
            const uint32_t tmem_tile = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)acc * 256u;
#pragma unroll 1
            for (int c0 = 32 * set; c0 < t.width; c0 += 64) {
                uint32_t r[32];
                tmem_ld32(tmem_tile + (uint32_t)c0, r);
                tmem_ld_wait();
                // Of two columns a lane keeps one and gives the other to its neighbour: even lanes end up
                // with both weight rows of column q, odd lanes with those of q + 1. The values of a chunk are
                // computed before any is stored: a branch around each one would leave nothing to hide the division behind.
                uint32_t v[16];
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    const float keep = __uint_as_float(odd ? r[2 * q + 1] : r[2 * q]);
                    const float got = __shfl_xor_sync(0xffffffffu, __uint_as_float(odd ? r[2 * q] : r[2 * q + 1]), 1);
                    const float lo = odd ? got : keep, hi = odd ? keep : got;
                    v[q] = EPI == 0 ? pack2(lo, hi) : __float_as_uint(pair_act<EPI>(lo, hi, act));
                }
                const int c = c0 + (odd ? 1 : 0);
                qi::bf16* o = out + (size_t)(t.row0 + c) * ld_out + (EPI == 0 ? n : n >> 1);
                if (n < N) {
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        if (c + 2 * q < t.rows) {
                            if (EPI == 0) *reinterpret_cast<uint32_t*>(o) = v[q];
                            else *o = __float2bfloat16_rn(__uint_as_float(v[q]));
                        }
                        o += 2 * ld_out;
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(acc_empty_bar(acc));
        }
    }
    tc_fence_before();
    cluster_sync_all();       // neither CTA goes before its partner is done with what it holds
    if (warp == 1 && *abort_flag) settle_in_flight();
    QI_TL_END(30 + EPI);
    if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

// Adds split-K partial sums in split order: out[i] = sum_s partial[s, i].
template <typename TOut>
__global__ void splitk_reduce_kernel(const float* __restrict__ partial, TOut* __restrict__ out, size_t n, int splits) {
    qi::pdl_enter();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float s = 0.f;
#pragma unroll 4
        for (int k = 0; k < splits; ++k) s += partial[(size_t)k * n + i];
        store1<TOut>(out + i, s);
    }
}

template <int BN, int STAGES, bool SWAP, typename TOut, int EPI>
int launch(const CUtensorMap& ma, const CUtensorMap& mb, TOut* out, int rows_a, int rows_b, int K, long long ld,
           int splits, int kb_per_split, long long split_stride, int* status, cudaStream_t stream,
           const RopeEpilogue& rope = RopeEpilogue{}) {
    auto kern = gemm_tcgen05_kernel<BN, STAGES, SWAP, TOut, EPI>;
    constexpr int smem = Smem<BN, STAGES>::kTotal;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return qi::fail("gemm_bf16: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured = true;
    }
    const long long tiles = (long long)((rows_a + BM - 1) / BM) * ((rows_b + BN - 1) / BN) * splits;
    // as many CTAs as fit on the GPU at once (by shared memory); each walks its share of the tiles
    const int per_sm = (227 * 1024) / smem > 0 ? (227 * 1024) / smem : 1;
    const long long resident = (long long)sm_count() * per_sm;
    const unsigned grid = (unsigned)(tiles < resident ? tiles : resident);
    qi::launch(kern, dim3(grid), dim3(kThreads), smem, stream, ma, mb, out, rows_a, rows_b, K, ld, kb_per_split, splits,
               split_stride, status, rope);
    return qi::check_launch("gemm_bf16");
}

template <typename TOut, int EPI>
int launch_pair(const CUtensorMap& ma, const CUtensorMap& mb, TOut* out, int M, int N, int K, long long ld, int* status,
                cudaStream_t stream, const RopeEpilogue& rope = RopeEpilogue{}, int splits = 1, long long split_stride = 0) {
    auto kern = gemm_tcgen05_pair_kernel<TOut, EPI>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem);
        if (e != cudaSuccess) return qi::fail("gemm_bf16: cannot reserve %d bytes of shared memory: %s", kPairSmem, cudaGetErrorString(e));
        configured = true;
    }
    const long long tiles = (long long)((M + 2 * BM - 1) / (2 * BM)) * ((N + 255) / 256) * splits;
    const long long pairs = sm_count() / 2;
    const unsigned grid = 2u * (unsigned)(tiles < pairs ? tiles : pairs);
    const int kb_total = (K + BK - 1) / BK;
    qi::launch(kern, dim3(grid), dim3(kThreads), kPairSmem, stream, ma, mb, out, M, N, K, ld, (kb_total + splits - 1) / splits,
               splits, split_stride, status, rope);
    return qi::check_launch("gemm_bf16 (CTA pairs)");
}

template <int EPI>
int launch_grouped(const CUtensorMap& mw, const WideMaps& mx, qi::bf16* out, const int* offsets, int groups, int n_rows, int N, int K,
                   long long ld, int* status, cudaStream_t stream, const RopeEpilogue& act) {
    auto kern = gemm_tcgen05_grouped_kernel<EPI>;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmem);
        if (e != cudaSuccess) return qi::fail("gemm_bf16_grouped: cannot reserve %d bytes of shared memory: %s", kWideSmem, cudaGetErrorString(e));
        configured = true;
    }
    const long long tiles = ((long long)n_rows / 256 + (groups < n_rows ? groups : n_rows)) * ((N + 2 * BM - 1) / (2 * BM));   // at most
    const long long pairs = sm_count() / 2;
    qi::launch(kern, dim3(2u * (unsigned)(tiles < pairs ? tiles : pairs)), dim3(kWideThreads), kWideSmem, stream, mw, mx, out, offsets, groups,
               n_rows, N, K, ld, status, act);
    return qi::check_launch("gemm_bf16_grouped");
}

// Pipeline stages by tile width: as many as let two CTAs stay resident on an SM for the narrow
// tiles (6 of 18 KB, 5 of 20 KB, 4 of 24 KB: the first stages' weight tiles are requested before
// the kernel waits for its predecessor, so deeper is better while two CTAs fit), 6 for the
// 128-wide tile and 4 for the widest, one CTA an SM.
constexpr int stages_of(int bn) { return bn <= 16 ? 6 : bn == 32 ? 5 : bn == 128 ? 6 : 4; }

template <bool SWAP, typename TOut, int EPI = 0>
int launch_bn(int bn, const CUtensorMap& ma, const CUtensorMap& mb, TOut* out, int rows_a, int rows_b, int K,
              long long ld, int splits, int kb_per_split, long long split_stride, int* status, cudaStream_t stream,
              const RopeEpilogue& rope = RopeEpilogue{}) {
    switch (bn) {
        case 16: return launch<16, stages_of(16), SWAP, TOut, EPI>(ma, mb, out, rows_a, rows_b, K, ld, splits, kb_per_split, split_stride, status, stream, rope);
        case 32: return launch<32, stages_of(32), SWAP, TOut, EPI>(ma, mb, out, rows_a, rows_b, K, ld, splits, kb_per_split, split_stride, status, stream, rope);
        case 64: return launch<64, stages_of(64), SWAP, TOut, EPI>(ma, mb, out, rows_a, rows_b, K, ld, splits, kb_per_split, split_stride, status, stream, rope);
        case 128: return launch<128, stages_of(128), SWAP, TOut, EPI>(ma, mb, out, rows_a, rows_b, K, ld, splits, kb_per_split, split_stride, status, stream, rope);
        case 256: return launch<256, stages_of(256), SWAP, TOut, EPI>(ma, mb, out, rows_a, rows_b, K, ld, splits, kb_per_split, split_stride, status, stream, rope);
    }
    return qi::fail("gemm_bf16: no kernel for a tile width of %d", bn);
}

}  // namespace

// The orientation (0: tokens on the 128 rows, 1: weights on the 128 rows, 2: tokens on the rows of
// CTA pairs), tile width and K split `qi_gemm_bf16` uses when the caller does not say
// (allow_split 0: the caller needs the whole sum in one CTA, as the fused activation does).
//
// Up to 64 tokens the product is a weight stream: the weights are the 128-row operand, the
// tokens the narrow one, and K is split until about 148 CTAs pull weights.
// Above that, the candidates (tokens as the narrow operand in one tile of 128 or 256 while they
// fit; tokens as the 128-row operand with weight tiles of 256 or 128; K in 1 to 16 parts) are
// compared by a count of k blocks per SM: waves of CTAs x (k blocks of a CTA + 12 for its start
// and its epilogue) x the relative cost of a k block at that width, plus what the partial sums
// cost to write and to read again (at 5.5 TB/s, in units of a 128 x 256 k block = 0.27 us).
// Splitting K fills the SMs when there are few tiles (a 4096-wide product of 512 tokens has 64
// tiles of 128 x 256) and evens out a ragged last wave; its price grows with the tokens. The
// constants were fitted to a sweep of all candidates over 72 to 4,096 tokens at four layer
// shapes: the choice is within 1% of the best candidate on average, 10% at worst.
extern "C" int qi_gemm_bf16_plan(int M, int N, int K, int allow_split, int* swap, int* bn, int* splits) {
    const int kb_total = (K + BK - 1) / BK;
    int sw = 1, b = 256, sp = 1;
    if (M <= 64) {
        b = M <= 16 ? 16 : M <= 32 ? 32 : 64;
        const int tiles = (N + BM - 1) / BM;
        // enough CTAs to keep the weight stream busy on 148 SMs, at least 8 k blocks per split
        // (filling every resident slot with 6 or 9 splits was measured no faster than powers of two)
        while (allow_split && tiles * sp < 148 && sp * 2 <= 16 && kb_total / (sp * 2) >= 8) sp *= 2;
        sp = (kb_total + (kb_total + sp - 1) / sp - 1) / ((kb_total + sp - 1) / sp);      // none without work (129 k blocks: 15 parts of 9)
    } else {
        const int sms = sm_count();
        double best = 1e30;
        const int split_choices[8] = {1, 2, 3, 4, 6, 8, 12, 16};
        for (int cand = 0; cand < 3; ++cand) {
            // 0: tokens narrow, one tile; 1, 2: tokens in rows of 128, weight tiles of 256, 128
            if (cand == 0 && M > 256) continue;
            const int c_swap = cand == 0, c_bn = cand == 0 ? (M <= 128 ? 128 : 256) : cand == 1 ? 256 : 128;
            const int rows_a = c_swap ? N : M, rows_b = c_swap ? M : N;
            const double k_cost = (c_bn == 256 ? 1.0 : 0.65) * (c_swap ? 1.05 : 1.0);
            for (int si = 0; si < (allow_split ? 8 : 1); ++si) {
                const int s = split_choices[si];
                const int kbs = (kb_total + s - 1) / s;
                if (s > 1 && ((s - 1) * kbs >= kb_total || kbs < 8)) continue;
                const long long units = (long long)((rows_a + BM - 1) / BM) * ((rows_b + c_bn - 1) / c_bn) * s;
                const long long waves = (units + sms - 1) / sms;
                double cost = (double)waves * (kbs + 12) * k_cost;
                if (s > 1) cost += (double)s * M * N * 8.0 / 5.5e12 / 0.27e-6;
                if (cost < best * 0.999) {
                    best = cost;
                    sw = c_swap;
                    b = c_bn;
                    sp = s;
                }
            }
        }
        // pairs of CTAs on tiles of 256 x 256: a k block of a pair's tile takes what a k block
        // of a 128 x 256 tile takes on one SM, less the 13% the lighter load on L2 and shared memory gives
        const long long pair_tiles = (long long)((M + 2 * BM - 1) / (2 * BM)) * ((N + 255) / 256);
        for (int si = 0; si < (allow_split ? 8 : 1); ++si) {
            const int s = split_choices[si];
            const int kbs = (kb_total + s - 1) / s;
            if (s > 1 && ((s - 1) * kbs >= kb_total || kbs < 8)) continue;
            const long long waves = (pair_tiles * s + sms / 2 - 1) / (sms / 2);
            double cost = (double)waves * (kbs + 12) * 0.87;
            if (s > 1) cost += (double)s * M * N * 8.0 / 5.5e12 / 0.27e-6;
            if (cost < best * 0.999) {
                best = cost;
                sw = 2;
                b = 256;
                sp = s;
            }
        }
    }
    *swap = sw; *bn = b; *splits = sp;
    return 0;
}

// y[M, N] = x[M, K] . w[N, K]^T, bf16 operands, out bf16 or float32 (out_dtype).
// With splits > 1, `workspace` must hold splits * M * N floats.
// epilogue 1: w's rows come in (gate, up) pairs and out[M, N / 2] = silu(gate) * up (bf16, no split).
// out may be null with splits > 1: the partial sums stay in the workspace for the consumer.
// epilogue 3: the same pairs through g sigmoid(alpha g) (u + 1), g = min(gate, limit), u = clamp(up, -limit, limit).
// ldx: elements from one row of x to the next (a block of columns of wider rows; 0: K).
extern "C" int qi_gemm_bf16_ex(const void* x, long long ldx, const void* w, void* out, int out_dtype, int M, int N, int K,
                               int swap, int bn, int splits, int epilogue, float limit, float alpha, void* workspace,
                               int* status, cudaStream_t stream) {
    QI_REQUIRE(ldx == 0 || (ldx >= K && ldx % 8 == 0), "gemm_bf16: rows of x must lie a multiple of 8 elements apart, at least K");
    QI_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_bf16: bad sizes M=%d N=%d K=%d", M, N, K);
    QI_REQUIRE(K % 8 == 0, "gemm_bf16: K=%d must be a multiple of 8 (16-byte rows for TMA)", K);
    QI_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0, "gemm_bf16: operands must be 16-byte aligned");
    QI_REQUIRE(splits >= 1 && (splits == 1 || workspace), "gemm_bf16: split-K needs a workspace");
    QI_REQUIRE(out_dtype == qi::kF32 || out_dtype == qi::kBF16, "gemm_bf16: output type must be float32 or bfloat16");
    QI_REQUIRE(epilogue == 0 || ((epilogue == 1 || epilogue == 3) && splits == 1 && out_dtype == qi::kBF16 && N % 2 == 0 && out),
               "gemm_bf16: the fused activation needs bfloat16 output, an even N and no K split");
    RopeEpilogue glu{};
    glu.limit = limit; glu.alpha = alpha;
    const int kb_total = (K + BK - 1) / BK;
    const int kb_per_split = (kb_total + splits - 1) / splits;
    QI_REQUIRE((splits - 1) * kb_per_split < kb_total, "gemm_bf16: %d splits leave one without work (K=%d)", splits, K);
    if (swap == 2) {
        // pairs of CTAs: tokens on the rows (the width of a plan is not read)
        CUtensorMap pa, pb;
        if (make_map(&pa, x, M, K, BM, ldx)) return 1;
        if (make_map(&pb, w, N, K, BM)) return 1;
        if (splits > 1) {
            float* ws = (float*)workspace;
            if (int rc = launch_pair<float, 0>(pa, pb, ws, M, N, K, N, status, stream, RopeEpilogue{}, splits, (long long)M * N)) return rc;
            if (out) {
                const size_t n = (size_t)M * N;
                unsigned blocks = (unsigned)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
                if (out_dtype == qi::kF32) qi::launch(splitk_reduce_kernel<float>, dim3(blocks), dim3(256), 0, stream, (const float*)ws, (float*)out, n, splits);
                else qi::launch(splitk_reduce_kernel<qi::bf16>, dim3(blocks), dim3(256), 0, stream, (const float*)ws, (qi::bf16*)out, n, splits);
                return qi::check_launch("splitk_reduce");
            }
            return 0;
        }
        if (epilogue == 1) return launch_pair<qi::bf16, 1>(pa, pb, (qi::bf16*)out, M, N, K, N / 2, status, stream);
        if (epilogue == 3) return launch_pair<qi::bf16, 3>(pa, pb, (qi::bf16*)out, M, N, K, N / 2, status, stream, glu);
        if (out_dtype == qi::kF32) return launch_pair<float, 0>(pa, pb, (float*)out, M, N, K, N, status, stream);
        return launch_pair<qi::bf16, 0>(pa, pb, (qi::bf16*)out, M, N, K, N, status, stream);
    }
    const void* a = swap ? w : x;
    const void* b = swap ? x : w;
    const int rows_a = swap ? N : M, rows_b = swap ? M : N;
    QI_REQUIRE((long long)((rows_a + BM - 1) / BM) * ((rows_b + bn - 1) / bn) * splits < 2147483647LL, "gemm_bf16: too many tiles");
    CUtensorMap ma, mb;
    if (make_map(&ma, a, rows_a, K, BM, swap ? 0 : ldx)) return 1;
    if (make_map(&mb, b, rows_b, K, bn, swap ? ldx : 0)) return 1;
    const long long split_stride = (long long)M * N;
    int rc;
    if (splits > 1) {
        float* ws = (float*)workspace;
        rc = swap ? launch_bn<true, float>(bn, ma, mb, ws, rows_a, rows_b, K, N, splits, kb_per_split, split_stride, status, stream)
                  : launch_bn<false, float>(bn, ma, mb, ws, rows_a, rows_b, K, N, splits, kb_per_split, split_stride, status, stream);
        if (rc) return rc;
        if (out) {
            const size_t n = (size_t)M * N;
            unsigned blocks = (unsigned)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
            if (out_dtype == qi::kF32) qi::launch(splitk_reduce_kernel<float>, dim3(blocks), dim3(256), 0, stream, (const float*)ws, (float*)out, n, splits);
            else qi::launch(splitk_reduce_kernel<qi::bf16>, dim3(blocks), dim3(256), 0, stream, (const float*)ws, (qi::bf16*)out, n, splits);
            return qi::check_launch("splitk_reduce");
        }
        return 0;
    }
    if (epilogue == 1)
        return swap ? launch_bn<true, qi::bf16, 1>(bn, ma, mb, (qi::bf16*)out, rows_a, rows_b, K, N / 2, 1, kb_per_split, 0, status, stream)
                    : launch_bn<false, qi::bf16, 1>(bn, ma, mb, (qi::bf16*)out, rows_a, rows_b, K, N / 2, 1, kb_per_split, 0, status, stream);
    if (epilogue == 3)
        return swap ? launch_bn<true, qi::bf16, 3>(bn, ma, mb, (qi::bf16*)out, rows_a, rows_b, K, N / 2, 1, kb_per_split, 0, status, stream, glu)
                    : launch_bn<false, qi::bf16, 3>(bn, ma, mb, (qi::bf16*)out, rows_a, rows_b, K, N / 2, 1, kb_per_split, 0, status, stream, glu);
    if (out_dtype == qi::kF32)
        return swap ? launch_bn<true, float>(bn, ma, mb, (float*)out, rows_a, rows_b, K, N, 1, kb_per_split, 0, status, stream)
                    : launch_bn<false, float>(bn, ma, mb, (float*)out, rows_a, rows_b, K, N, 1, kb_per_split, 0, status, stream);
    return swap ? launch_bn<true, qi::bf16>(bn, ma, mb, (qi::bf16*)out, rows_a, rows_b, K, N, 1, kb_per_split, 0, status, stream)
                : launch_bn<false, qi::bf16>(bn, ma, mb, (qi::bf16*)out, rows_a, rows_b, K, N, 1, kb_per_split, 0, status, stream);
}

extern "C" int qi_gemm_bf16(const void* x, const void* w, void* out, int out_dtype, int M, int N, int K,
                            int swap, int bn, int splits, int epilogue, void* workspace, int* status,
                            cudaStream_t stream) {
    QI_REQUIRE(epilogue == 0 || epilogue == 1, "gemm_bf16: unknown epilogue %d", epilogue);
    return qi_gemm_bf16_ex(x, 0, w, out, out_dtype, M, N, K, swap, bn, splits, epilogue, 0.f, 0.f, workspace, status, stream);
}

// Group e's rows of x [rows, K] (offsets[e] .. offsets[e + 1] - 1, DEVICE memory [groups + 1], ascending) times w[e] [N, K], all
// bfloat16: out [rows, N], or [rows, N / 2] with an epilogue over the (gate, up) pairs of w's rows (1: silu(g) u; 3: the clamped
// form with limit and alpha). Rows of no group are not written.
extern "C" int qi_gemm_bf16_grouped(const void* x, const void* w, void* out, const int* offsets, int groups, int rows, int N, int K,
                                    int epilogue, float limit, float alpha, int* status, cudaStream_t stream) {
    QI_REQUIRE(groups > 0 && groups <= kWideMaxGroups && rows >= 0 && N > 0 && K > 0, "gemm_bf16_grouped: bad sizes groups=%d rows=%d N=%d K=%d", groups, rows, N, K);
    QI_REQUIRE(K % 8 == 0 && N % 2 == 0, "gemm_bf16_grouped: K=%d must be a multiple of 8 and N=%d even", K, N);
    QI_REQUIRE((((uintptr_t)x | (uintptr_t)w) & 15) == 0 && ((uintptr_t)out & 3) == 0, "gemm_bf16_grouped: operands must be 16-byte aligned, the result 4-byte aligned");
    QI_REQUIRE(epilogue == 0 || epilogue == 1 || epilogue == 3, "gemm_bf16_grouped: unknown epilogue %d", epilogue);
    QI_REQUIRE((long long)groups * N < 2147483647LL && ((long long)rows / 256 + groups) * ((N + 255) / 256) < 2147483647LL, "gemm_bf16_grouped: too many tiles");
    if (rows == 0) return 0;
    QI_REQUIRE(offsets, "gemm_bf16_grouped: the offsets are missing");
    CUtensorMap mw;
    WideMaps mx;
    if (make_map(&mw, w, groups * N, K, BM)) return 1;
    for (int i = 0; i < 8; ++i)
        if (make_map(&mx.of[i], x, rows, K, 16 * (i + 1))) return 1;
    RopeEpilogue act{};
    act.limit = limit; act.alpha = alpha;
    qi::bf16* o = (qi::bf16*)out;
    if (epilogue == 1) return launch_grouped<1>(mw, mx, o, offsets, groups, rows, N, K, N / 2, status, stream, act);
    if (epilogue == 3) return launch_grouped<3>(mw, mx, o, offsets, groups, rows, N, K, N / 2, status, stream, act);
    return launch_grouped<0>(mw, mx, o, offsets, groups, rows, N, K, N, status, stream, act);
}

// The q/k/v projection of many tokens with what follows it fused into the epilogue:
// [q | k | v] = x[M, K] . w[(nq + 2 nkv) * 128, K]^T, then RMSNorm of every query and key head
// (gains null: none), the half-split rotation by the token's position (cos_t null: none), queries
// to q_out [M, nq * 128], keys and values to the paged cache (k_pages null: not written). Head size
// 128, rotation over the whole head, bfloat16 throughout. The operands are not swapped, so this is
// the path for prompts; few tokens go through qi_gemm_bf16 (K split) and qi_qk_norm_rope_kv.
extern "C" int qi_gemm_bf16_qkv_rope(const void* x, const void* w, int M, int K, void* q_out, const float* q_gain,
                                     const float* k_gain, float eps, const float* cos_t, const float* sin_t,
                                     int table_positions, const int* positions, const int* token_req,
                                     const int* block_table, int max_blocks, int page_size, int num_pages,
                                     void* k_pages, void* v_pages, int nq, int nkv, int* status, cudaStream_t stream) {
    QI_REQUIRE(M > 0 && K > 0 && nq > 0 && nkv > 0, "gemm_bf16_qkv_rope: bad sizes M=%d K=%d heads %d/%d", M, K, nq, nkv);
    QI_REQUIRE(K % 8 == 0, "gemm_bf16_qkv_rope: K=%d must be a multiple of 8 (16-byte rows for TMA)", K);
    QI_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)w & 15) == 0 && ((uintptr_t)q_out & 15) == 0 &&
               ((uintptr_t)k_pages & 15) == 0 && ((uintptr_t)v_pages & 15) == 0,
               "gemm_bf16_qkv_rope: operands, q_out and pages must be 16-byte aligned");
    QI_REQUIRE(q_out && positions, "gemm_bf16_qkv_rope: q_out and positions are needed");
    QI_REQUIRE((cos_t == nullptr) == (sin_t == nullptr) && (!cos_t || table_positions > 0), "gemm_bf16_qkv_rope: incomplete rotation table");
    QI_REQUIRE(((uintptr_t)cos_t & 15) == 0 && ((uintptr_t)sin_t & 15) == 0 && ((uintptr_t)q_gain & 15) == 0 && ((uintptr_t)k_gain & 15) == 0,
               "gemm_bf16_qkv_rope: gains and tables must be 16-byte aligned");
    QI_REQUIRE((k_pages == nullptr) == (v_pages == nullptr), "gemm_bf16_qkv_rope: k and v pages must come together");
    QI_REQUIRE(!k_pages || (page_size > 0 && max_blocks > 0 && num_pages > 0 && block_table && token_req),
               "gemm_bf16_qkv_rope: incomplete page arguments");
    const long long n_ll = (long long)(nq + 2 * nkv) * 128;
    QI_REQUIRE(n_ll < 2147483647LL, "gemm_bf16_qkv_rope: too many heads");
    const int N = (int)n_ll;
    int plan_mode, bn, plan_splits;
    qi_gemm_bf16_plan(M > 256 ? M : 257, N, K, 0, &plan_mode, &bn, &plan_splits);   // the width for operands that are not swapped
    if (bn < 128) bn = 128;                                                        // a tile holds whole heads
    const int kb_total = (K + BK - 1) / BK;
    QI_REQUIRE((long long)((M + BM - 1) / BM) * ((N + bn - 1) / bn) < 2147483647LL, "gemm_bf16_qkv_rope: too many tiles");
    CUtensorMap ma, mb;
    if (make_map(&ma, x, M, K, BM)) return 1;
    if (make_map(&mb, w, N, K, bn)) return 1;
    RopeEpilogue e;
    e.q_out = (qi::bf16*)q_out; e.q_gain = q_gain; e.k_gain = k_gain; e.cos_t = cos_t; e.sin_t = sin_t;
    e.positions = positions; e.token_req = token_req; e.block_table = block_table;
    e.k_pages = (qi::bf16*)k_pages; e.v_pages = (qi::bf16*)v_pages; e.eps = eps;
    e.max_blocks = max_blocks; e.page_size = page_size; e.num_pages = num_pages; e.nq = nq; e.nkv = nkv;
    e.table_positions = table_positions;
    if (plan_mode == 2) {
        CUtensorMap pb;
        if (make_map(&pb, w, N, K, BM)) return 1;
        return launch_pair<qi::bf16, 2>(ma, pb, (qi::bf16*)nullptr, M, N, K, N, status, stream, e);
    }
    if (bn == 256)
        return launch<256, stages_of(256), false, qi::bf16, 2>(ma, mb, (qi::bf16*)nullptr, M, N, K, N, 1, kb_total, 0, status, stream, e);
    return launch<128, stages_of(128), false, qi::bf16, 2>(ma, mb, (qi::bf16*)nullptr, M, N, K, N, 1, kb_total, 0, status, stream, e);
}


QI_TL_EXPORT(qi_timeline_gemm)
