// The product of the 32-bit path at the sizes of real models: y[M, N] = x[M, K] . w[N, K]^T with every operand's 24 bits on the
// tensor cores.
//
// A 32-bit number is the sum of three bfloat16 numbers, h + m + l: each is the rounding of what the ones before it leave, the
// remainders are exact in 32 bits, and 8 bits each make 24 (below 2^-110 the last part meets the smallest bfloat16 number, 2^-133: such
// numbers keep fewer bits beside larger ones of their row, from 2^24 times as large on, and all of them in a row that holds no larger one).
// bfloat16 products are exact in 32 bits, so
//     x w = hh + (hm + mh) + (hl + mm + lh)        and what is left out (ml, lm, ll) is below 2^-25 of the product.
// Six tcgen05 MMAs (kind::f16, 32-bit accumulation) over 64 k make a chunk; they start from zero, the five small terms first, so that
// the sum in tensor memory is short and its roundings are those of a 64th of the whole at K = 4,096. The chunks are added
// in registers, to nearest, k ascending. Error against 64 bits, in 2-norms: 1.0e-7 to 1.2e-7 from K = 1,024 to 8,192 (the chain of
// single FMAs that gemm_simt.cu computes: 5.7e-7 to 1.6e-6).
//
// A row's result depends on neither the number of rows nor the other rows: the cut of K depends on N and K alone. A row of x or w that
// holds an infinity, a NaN or a number that rounds to infinity as a bfloat16, or nothing from 2^-86 up beside zeros, is flagged on the way.
// Its results, and every one whose sum here is not finite (parts of finite operands may overflow where the sum does not, and an infinite
// h h meets infinities of both signs in the small terms), are computed by the chain of FMAs over all of K instead: they are what that
// makes of them, bit for bit.
//
// A CTA computes 128 rows of w x up to 128 tokens (the tokens cut evenly, in steps of 16) over its part of K. Roles (18 warps):
//   warp 0       TMA: the tokens' three parts, cut beforehand by split_rows_kernel (tokens are few, weights are not), and the
//                request for the weights' tiles to come to the L2, eight chunks ahead
//   warp 1       MMA
//   warps 2-9    add a chunk's accumulator to registers while the next chunk is computed in the other half of tensor memory
//   warps 10-17  read w (32-bit, up to two chunks of 32 KB ahead in registers, from the L2), cut it, and write the three
//                tiles to shared memory in the layout of the 128-byte swizzle
// Two stages of both operands' parts fill the shared memory (192 KB). What bounds a chunk is the way of a stage from the converting
// warps through the MMAs and back, 1.2 us for one token and 1.4 for 100: leaving out the conversion, the loads or most MMAs (24 of
// 70 cycles each, 0.9 us, run beside the next stage's conversion), one at a time, saved under 10%. Waits are bounded as in gemm_tcgen05.cu.
// Measured against the chain of FMAs, one token and 201: [4096, 4096] 87 -> 37 and 270 -> 68 us; [24576, 4096] 325 -> 143 and
// 1,166 -> 292 us; [4096, 12288] 255 -> 75 and 805 -> 154 us.
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int kSplitThreads = 576;
constexpr int kTileBytes = 128 * BK * 2;                 // one part of 128 rows x 64 k
constexpr int kPartStage = 3 * kTileBytes;               // h, m, l
constexpr int kSplitBars = 4 * kPartStage;               // two stages of w's parts, two of x's
constexpr int kSplitSmem = kSplitBars + 8 * 10 + 16 + 128 * 4 + 1024;
constexpr int kAhead = 8;                                // chunks from the request for a tile of w to its use

__device__ __forceinline__ void prefetch_2d(const CUtensorMap* map, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}

// The three parts of two neighbours: packed pairs, the first number in the low half.
__device__ __forceinline__ void cut2(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    const __nv_bfloat162 hv = __floats2bfloat162_rn(a, b);
    h = *reinterpret_cast<const uint32_t*>(&hv);
    const float ra = a - __uint_as_float(h << 16), rb = b - __uint_as_float(h & 0xffff0000u);
    const __nv_bfloat162 mv = __floats2bfloat162_rn(ra, rb);
    m = *reinterpret_cast<const uint32_t*>(&mv);
    const __nv_bfloat162 lv = __floats2bfloat162_rn(ra - __uint_as_float(m << 16), rb - __uint_as_float(m & 0xffff0000u));
    l = *reinterpret_cast<const uint32_t*>(&lv);
}

// The largest magnitude of a row, number by number; a NaN stays.
__device__ __forceinline__ float largest(float top, float a, float b) {
    float d;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(top), "f"(a), "f"(b));
    return d;
}
// Whether a row with this largest magnitude goes through the chain of FMAs. (The first bound: half a step of bfloat16 below 2^128.)
__device__ __forceinline__ bool needs_chain(float top) { return !(top < 3.3961775e38f) || (top != 0.f && top < 0x1p-86f); }

__device__ __forceinline__ float chain(const float* __restrict__ x, const float* __restrict__ w, int K) {
    float v = 0.f;
#pragma unroll 4
    for (int k = 0; k < K; ++k) v = fmaf(x[k], w[k], v);
    return v;
}

// parts [3, M, K] of x [M, K]; flags[row] = 1 when the row needs the chain. One block a row, K a multiple of 4.
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ x, qi::bf16* __restrict__ parts, int* __restrict__ flags, int M, int K) {
    qi::pdl_enter();
    const size_t row = blockIdx.x;
    const float4* src = reinterpret_cast<const float4*>(x + row * K);
    uint2* dst = reinterpret_cast<uint2*>(parts + row * K);
    const size_t part = (size_t)M * K / 4;
    float top = 0.f;
    for (int i = threadIdx.x; i < K / 4; i += 256) {
        const float4 v = src[i];
        uint2 h, m, l;
        cut2(v.x, v.y, h.x, m.x, l.x);
        cut2(v.z, v.w, h.y, m.y, l.y);
        top = largest(largest(top, v.x, v.y), v.z, v.w);
        dst[i] = h;
        dst[part + i] = m;
        dst[2 * part + i] = l;
    }
    const int huge = __syncthreads_or(!(top < 3.3961775e38f)), some = __syncthreads_or(top != 0.f), real = __syncthreads_or(top >= 0x1p-86f);
    if (threadIdx.x == 0) flags[row] = huge || (some && !real);
}

__global__ void __launch_bounds__(kSplitThreads)
gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const float* __restrict__ x,
                      const float* __restrict__ w, float* __restrict__ out, const int* __restrict__ x_flags, int M, int N, int K,
                      int width, int tiles_t, int chunks_per_split, int* __restrict__ status) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* aligned = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t bars = base + kSplitBars;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aligned + kSplitBars + 8 * 10);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* w_top = reinterpret_cast<int*>(tmem_slot + 4);                 // [128]: the largest magnitudes of the rows' parts (as bits, which order as the numbers do)
    auto a_full = [&](int s) { return bars + 8u * s; };
    auto b_full = [&](int s) { return bars + 8u * (2 + s); };
    auto empty = [&](int s) { return bars + 8u * (4 + s); };
    auto acc_full = [&](int a) { return bars + 8u * (6 + a); };
    auto acc_empty = [&](int a) { return bars + 8u * (8 + a); };
    auto a_tile = [&](int s) { return base + (uint32_t)s * kPartStage; };
    auto b_tile = [&](int s) { return base + (uint32_t)(2 + s) * kPartStage; };

    qi::pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // token tiles first: CTAs that read the same weights run together
    const int tile_t = blockIdx.x % tiles_t, n0 = (blockIdx.x / tiles_t) * 128, t0 = tile_t * width;
    const int chunk0 = blockIdx.y * chunks_per_split, chunks = min(K / BK - chunk0, chunks_per_split);
    out += (size_t)blockIdx.y * M * N;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(a_full(s), 8);        // one arrival a converting warp
            mbar_init(b_full(s), 1);
            mbar_init(empty(s), 1);
            mbar_init(acc_full(s), 1);
            mbar_init(acc_empty(s), 8);     // one arrival an adding warp
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < 128) w_top[threadIdx.x] = 0;
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 256);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- the tokens' parts ----------------
        if (lane == 0) {
            for (int c = 2; c < kAhead && c < chunks; ++c) prefetch_2d(&map_w, (chunk0 + c) * BK, n0);     // (the first two are read at once)
            qi::pdl_wait();
            for (int c = 0; c < chunks; ++c) {
                const int s = c & 1;
                if (c + kAhead < chunks) prefetch_2d(&map_w, (chunk0 + c + kAhead) * BK, n0);
                if (!mbar_wait(empty(s), ((uint32_t)(c >> 1) & 1u) ^ 1u, abort_flag, status)) {
                    give_up(abort_flag, status);
                    break;
                }
                mbar_expect_tx(b_full(s), 3u * (uint32_t)width * BK * 2);
                for (int p = 0; p < 3; ++p)
                    tma_load_2d(b_tile(s) + p * kTileBytes, &map_x, b_full(s), (chunk0 + c) * BK, p * M + t0);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA ----------------
        if (lane == 0) {
            qi::pdl_wait();
            const uint32_t idesc = make_idesc(128, width);
            for (int c = 0; c < chunks; ++c) {
                const int s = c & 1;
                const uint32_t parity = (uint32_t)(c >> 1) & 1u;
                if (!mbar_wait(acc_empty(s), parity ^ 1u, abort_flag, status) || !mbar_wait(b_full(s), parity, abort_flag, status) ||
                    !mbar_wait(a_full(s), parity, abort_flag, status)) {
                    give_up(abort_flag, status);
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)s * 128u;
                constexpr int kTerms[6][2] = {{2, 0}, {0, 2}, {1, 1}, {1, 0}, {0, 1}, {0, 0}};      // (part of w, part of x), small ones first
#pragma unroll
                for (int p = 0; p < 6; ++p) {
                    const uint64_t adesc = make_smem_desc(a_tile(s) + kTerms[p][0] * kTileBytes);
                    const uint64_t bdesc = make_smem_desc(b_tile(s) + kTerms[p][1] * kTileBytes);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) umma_bf16(d, adesc + 2u * k, bdesc + 2u * k, idesc, (p > 0 || k > 0) ? 1u : 0u);
                }
                umma_commit(empty(s));
                umma_commit(acc_full(s));
            }
        }
    } else if (warp < 10) {
        // ---------------- sums ----------------
        const int quarter = warp & 3, set = (warp - 2) >> 2;
        const int groups = width / 16, first = set ? (groups + 1) / 2 : 0, last = set ? groups : (groups + 1) / 2;   // of 16 tokens, at most four
        float acc[4][16];
#pragma unroll
        for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[g][i] = 0.f;
        bool ok = true;
        qi::pdl_wait();           // (every bounded wait counts from the end of the kernel before)
        if (threadIdx.x == 64 && failed_before(status)) give_up(abort_flag, status);
        for (int c = 0; c < chunks; ++c) {
            const int s = c & 1;
            if (!mbar_wait_warp(acc_full(s), (uint32_t)(c >> 1) & 1u, abort_flag, status)) {
                if (lane == 0) give_up(abort_flag, status);
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t addr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)s * 128u + 16u * first;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                if (first + g < last) {
                    uint32_t r[32];
                    tmem_ld16(addr + 16u * g, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[g][i] += __uint_as_float(r[i]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(s));
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");      // the converting warps have left their rows' magnitudes
        const int row = quarter * 32 + lane, n = n0 + row, count = 16 * (last - first), tf = t0 + 16 * first;
        // a lane looks at two tokens' flags: looked up where a value is stored, each would cost its latency in turn
        const bool x_any = (lane < count && tf + lane < M && x_flags[tf + lane]) || (lane + 32 < count && tf + lane + 32 < M && x_flags[tf + lane + 32]);
        bool again = needs_chain(__int_as_float(w_top[row]));
        const bool w_bad = again;
        again |= __any_sync(0xffffffffu, x_any);
        if (ok && n < N) {
#pragma unroll
            for (int g = 0; g < 4; ++g)
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int t = tf + 16 * g + i;
                    if (first + g < last && t < M) {
                        out[(size_t)t * N + n] = acc[g][i];
                        again |= !(fabsf(acc[g][i]) <= 3.402823466e38f);
                    }
                }
        }
        if (ok && n < N && again) {
            // with K in parts none of them can tell what the chain makes of all: a NaN asks for it where they are added
#pragma unroll 1
            for (int i = 0; i < count && tf + i < M; ++i) {
                float* place = out + (size_t)(tf + i) * N + n;
                if (!w_bad && !x_flags[tf + i] && fabsf(*place) <= 3.402823466e38f) continue;
                *place = gridDim.y > 1 ? __int_as_float(0x7fffffff) : chain(x + (size_t)(tf + i) * K, w + (size_t)n * K, K);
            }
        }
    } else {
        // ---------------- the weights' parts ----------------
        const int tid = threadIdx.x - 320;
        const int k4 = (tid & 15) * 4, r0 = tid >> 4;          // this thread's 4 k of rows r0, r0 + 16, ...
        float4 ring[2][8];
        float top[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) top[i] = 0.f;
        const float* src = w + (size_t)(n0 + r0) * K + (size_t)chunk0 * BK + k4;
        const size_t step = (size_t)16 * K;
        auto fetch = [&](int c, float4 (&v)[8]) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                v[i] = (c < chunks && n0 + r0 + 16 * i < N) ? __ldg(reinterpret_cast<const float4*>(src + i * step + (size_t)c * BK)) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        // the 16-byte pieces of a row of 128 bytes are permuted by the row's place in its group of eight
        const uint32_t place = (uint32_t)r0 * 128u + ((((uint32_t)k4 >> 3) ^ ((uint32_t)r0 & 7u)) << 4) + (((uint32_t)k4 >> 2) & 1u) * 8u;
        fetch(0, ring[0]);       // no kernel of a step writes weights: these need not wait for the kernel before
        fetch(1, ring[1]);
        qi::pdl_wait();
        auto chunk = [&](int c, float4 (&v)[8]) -> bool {
            const int s = c & 1;
            if (!mbar_wait_warp(empty(s), ((uint32_t)(c >> 1) & 1u) ^ 1u, abort_flag, status)) {
                if (lane == 0) give_up(abort_flag, status);
                return false;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                uint2 h, m, l;
                cut2(v[i].x, v[i].y, h.x, m.x, l.x);
                cut2(v[i].z, v[i].w, h.y, m.y, l.y);
                top[i] = largest(largest(top[i], v[i].x, v[i].y), v[i].z, v[i].w);
                const uint32_t dst = a_tile(s) + place + (uint32_t)i * 2048u;      // 16 rows further (the same place in their group of eight)
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst), "r"(h.x), "r"(h.y) : "memory");
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + kTileBytes), "r"(m.x), "r"(m.y) : "memory");
                asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + 2 * kTileBytes), "r"(l.x), "r"(l.y) : "memory");
            }
            fetch(c + 2, v);
            if (c + 1 == chunks) {
#pragma unroll
                for (int i = 0; i < 8; ++i) atomicMax(&w_top[r0 + 16 * i], __float_as_int(top[i]) & 0x7fffffff);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the MMA reads through the async proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(a_full(s));
            return true;
        };
        for (int c = 0; c < chunks; c += 2) {
            if (!chunk(c, ring[0])) break;
            if (c + 1 < chunks && !chunk(c + 1, ring[1])) break;
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1 && *abort_flag) settle_in_flight();
    if (warp == 1) tmem_dealloc(tmem_base, 256);
}

// out = the parts of K added in order; the chain where that is not finite.
__global__ void __launch_bounds__(256)
add_parts_kernel(const float4* __restrict__ parts, float4* __restrict__ out, size_t n4, int splits, const float* __restrict__ x,
                 const float* __restrict__ w, int N, int K) {
    qi::pdl_enter();
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n4; i += (size_t)gridDim.x * 256) {
        float4 s = parts[i];
#pragma unroll 4
        for (int k = 1; k < splits; ++k) {
            const float4 v = parts[k * n4 + i];
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        if (!(largest(largest(0.f, s.x, s.y), s.z, s.w) <= 3.402823466e38f)) {
            const size_t t = i * 4 / N, n = i * 4 - t * N;          // (N is a multiple of 4: four columns of one row)
            float* v = &s.x;
#pragma unroll 1
            for (int j = 0; j < 4; ++j)
                if (!(fabsf(v[j]) <= 3.402823466e38f)) v[j] = chain(x + t * K, w + (n + j) * K, K);
        }
        out[i] = s;
    }
}

// Parts of K: by N and K alone, so that a row's sums do not depend on how many rows there are. The count, from 1 to 12 and with at least
// eight chunks of 64 each, that leaves the fewest chunks to the fullest SM; 6 more for a CTA's start and end.
int parts_of_k(int N, int K) {
    const int tiles = (N + 127) / 128, chunks = K / BK;
    int best = 1;
    long long least = -1;
    for (int s = 1; s <= 12; ++s) {
        const int each = (chunks + s - 1) / s;
        if (s > 1 && (each < 8 || (s - 1) * each >= chunks)) continue;
        const long long cost = ((long long)tiles * s + 147) / 148 * (each + 6);
        if (least < 0 || cost < least) { least = cost; best = s; }
    }
    return best;
}

size_t round256(size_t n) { return (n + 255) & ~(size_t)255; }

// Rows of x that go through the workspace at a time: the partial sums of a long prompt would take gigabytes (8,001 rows by 24,576
// columns in 3 parts: 2.4 GB), and eight tiles of tokens already share every tile of weights that comes from HBM.
constexpr int kRowsAtOnce = 1024;

int run_rows(const float* x, const float* w, float* y, int M, int N, int K, void* workspace, const CUtensorMap& mw, int* status, cudaStream_t stream) {
    qi::bf16* parts = (qi::bf16*)workspace;
    int* flags = (int*)((char*)workspace + round256((size_t)3 * M * K * 2));
    float* sums = (float*)((char*)flags + round256((size_t)M * 4));
    const int splits = parts_of_k(N, K), each = (K / BK + splits - 1) / splits;
    const int tiles_t = (M + 127) / 128, width = ((M + tiles_t - 1) / tiles_t + 15) & ~15;
    const long long tiles = (long long)((N + 127) / 128) * tiles_t;
    QI_REQUIRE(tiles < 2147483647LL, "gemm_f32: too many tiles");
    CUtensorMap mx;
    if (make_map(&mx, parts, 3 * M, K, width)) return 1;
    qi::launch(split_rows_kernel, dim3(M), dim3(256), 0, stream, x, parts, flags, M, K);
    if (int rc = qi::check_launch("split_rows")) return rc;
    qi::launch(gemm_f32_split_kernel, dim3((unsigned)tiles, splits), dim3(kSplitThreads), kSplitSmem, stream, mx, mw, x, w, splits > 1 ? sums : y,
               (const int*)flags, M, N, K, width, tiles_t, each, status);
    if (int rc = qi::check_launch("gemm_f32_split")) return rc;
    if (splits > 1) {
        const size_t n4 = (size_t)M * N / 4;
        const size_t blocks = (n4 + 255) / 256;
        qi::launch(add_parts_kernel, dim3((unsigned)(blocks < 148 * 8 ? blocks : 148 * 8)), dim3(256), 0, stream, (const float4*)sums, (float4*)y, n4, splits, x, w, N, K);
        return qi::check_launch("add_parts");
    }
    return 0;
}

}  // namespace

// Bytes of workspace that qi_gemm_f32 needs for a product of these sizes; 0: it takes gemm_simt.cu's kernel, which needs none.
// The line: below 2^22 weights (16 MB) both are a matter of latency and the FMA kernel, one launch instead of two or three, is the faster one.
extern "C" long long qi_gemm_f32_workspace(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0 || K % BK || N % 4 || (long long)N * K < (1LL << 22)) return 0;
    const int splits = parts_of_k(N, K);
    if (M > kRowsAtOnce) M = kRowsAtOnce;
    return (long long)(round256((size_t)3 * M * K * 2) + round256((size_t)M * 4) + (splits > 1 ? (size_t)splits * M * N * 4 : 0));
}

extern "C" int qi_gemm_f32_fma(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream);

// y[M, N] = x[M, K] . w[N, K]^T, all float32, rows one after the other; w are weights, which no kernel in flight writes: their first rows are
// read ahead of the stream's order. workspace: qi_gemm_f32_workspace(M, N, K) bytes, 256-byte
// aligned (null where that is 0).
extern "C" int qi_gemm_f32(const float* x, const float* w, float* y, int M, int N, int K, void* workspace, int* status,
                           cudaStream_t stream) {
    QI_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    if (M == 0) return 0;
    if (!workspace || qi_gemm_f32_workspace(M, N, K) == 0 || (((uintptr_t)x | (uintptr_t)w | (uintptr_t)y) & 15))
        return qi_gemm_f32_fma(x, w, y, M, N, K, stream);
    QI_REQUIRE(((uintptr_t)workspace & 15) == 0, "gemm_f32: the workspace must be 16-byte aligned");
    CUtensorMap mw;
    {
        EncodeTiledFn enc = get_encode();
        if (!enc) return qi::fail("gemm_f32: cuTensorMapEncodeTiled is not available from the driver");
        const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N}, strides[1] = {(cuuint64_t)K * 4};
        const cuuint32_t box[2] = {(cuuint32_t)BK, 128}, estr[2] = {1, 1};
        const CUresult r = enc(&mw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(w), dims, strides, box, estr,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return qi::fail("gemm_f32: cuTensorMapEncodeTiled failed with code %d (N=%d K=%d)", (int)r, N, K);
    }
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(gemm_f32_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmem) != cudaSuccess)
            return qi::fail("gemm_f32: %d bytes of shared memory were refused", kSplitSmem);
        configured = true;
    }
    for (int r = 0; r < M; r += kRowsAtOnce)
        if (int rc = run_rows(x + (size_t)r * K, w, y + (size_t)r * N, M - r < kRowsAtOnce ? M - r : kRowsAtOnce, N, K, workspace, mw, status, stream)) return rc;
    return 0;
}
