// Plain matrix product on the 32-bit FMA pipe: y[M, N] = x[M, K] . w[N, K]^T.
//
// `w` is in the checkpoint's [out, in] layout, so both operands are read along
// K. Any element type for x, w and y; products and sums are 32-bit, and every
// output element is accumulated by one thread with k ascending, so a row's
// result does not depend on which other rows are in the batch (nor on which of
// the two kernels below computes it). This is the
// matrix product of the true 32-bit path (no tensor cores, no TF32) and of
// any operand combination the tensor-core kernel does not take. The reference
// computes out[c] = sum_k x[k] * W[k, c] with k ascending
// (backends/cpu/src/matmul.rs:50-59).
//
// gemm_f32_kernel    32-bit x, w and y in rows of whole 16-byte pieces: the 32-bit path itself
// gemm_simt_kernel   everything else, one element at a time
#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TX, typename TW, typename TY>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TX* __restrict__ x, const TW* __restrict__ w, TY* __restrict__ y, int M,
                 int N, int K, long long ldx, long long ldw, long long ldy, long long sx, long long sw,
                 long long sy) {
    __shared__ float xs[BK][BM + 4];
    __shared__ float ws[BK][BN + 4];
    qi::pdl_enter();
    x += (size_t)blockIdx.z * sx;      // a batch of products: one operand set per grid.z
    w += (size_t)blockIdx.z * sw;
    y += (size_t)blockIdx.z * sy;
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;  // tx over N, ty over M
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;

    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    // Each thread loads 4 consecutive k of one row of each tile.
    const int lrow = tid / 4;        // 0..63
    const int lk = (tid % 4) * 4;    // 0,4,8,12
    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lk + i;
            float a = 0.f, b = 0.f;
            if (k < K) {
                if (m0 + lrow < M) a = qi::to_f32<TX>(x[(size_t)(m0 + lrow) * ldx + k]);
                if (n0 + lrow < N) b = qi::to_f32<TW>(w[(size_t)(n0 + lrow) * ldw + k]);
            }
            xs[lk + i][lrow] = a;
            ws[lk + i][lrow] = b;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = xs[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = ws[k][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n < N) y[(size_t)m * ldy + n] = qi::from_f32<TY>(acc[i][j]);
        }
    }
}

template <typename TX, typename TW, typename TY>
int launch(const void* x, const void* w, void* y, int M, int N, int K, long long ldx,
           long long ldw, long long ldy, cudaStream_t stream, int batch = 1, long long sx = 0, long long sw = 0,
           long long sy = 0) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    qi::launch(gemm_simt_kernel<TX, TW, TY>, grid, dim3(256), 0, stream, (const TX*)x, (const TW*)w, (TY*)y, M, N, K, ldx, ldw,
               ldy, sx, sw, sy);
    return qi::check_launch("gemm_simt");
}

// ---- the 32-bit path
//
// Bound by the FMA pipe for prompts (128 results a clock and SM), by latency below about 60 rows. 256 threads
// are 16 x 16; a thread owns TM rows (16 apart) and TN columns (16 apart) of the tile. Both operands are
// copied by cp.async in their own layout, 32 k of every row a stage, rows padded to 36 floats: a 16-byte
// read of 8 neighbouring rows then touches every bank once. A thread reads four k of its rows and
// columns at a time, TM + TN 16-byte reads for 4 TM TN multiply-adds; the k chain of an element stays in
// order. Small tiles have up to eight stages in flight. With `ahead` the first stages' weights are requested before the wait
// for the kernel before this one: for callers whose w no kernel in flight writes.
// Measured, [201, 4096] . [24576, 4096]^T: 2,090 us with the kernel above, 1,168 us with this one (62% of the
// FMA pipe's cycles, 72% of the issue slots); [201, 12288] . [4096, 12288]^T: 1,650 and 808 us. Packed FMAs
// (fma.rn.f32x2) over a transposed copy were no faster (1,330 us): they take two cycles of the same pipe.
constexpr int FK = 32, FS = FK + 4;        // k of a stage; floats from one row of a stage to the next

constexpr int f32_stage_bytes(int tm, int tn) { return 16 * (tm + tn) * FS * 4; }
constexpr int f32_stages(int tm, int tn) {
    const int n = 110 * 1024 / f32_stage_bytes(tm, tn);
    return n > 8 ? 8 : n;
}

__device__ __forceinline__ void copy16(uint32_t dst, const float* src, bool real) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(real ? 16 : 0) : "memory");
}

template <int TM, int TN>
__global__ void __launch_bounds__(256, TM * TN >= 16 ? 2 : 3)
gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K,
                long long ldx, long long ldw, long long ldy, long long sx, long long sw, long long sy, int ahead) {
    constexpr int TILE_M = 16 * TM, TILE_N = 16 * TN, STAGES = f32_stages(TM, TN), STAGE = (TILE_M + TILE_N) * FS;
    extern __shared__ __align__(16) float f32_smem[];
    qi::pdl_launch_dependents();
    x += (size_t)blockIdx.z * sx;
    w += (size_t)blockIdx.z * sw;
    y += (size_t)blockIdx.z * sy;
    const int tiles_m = (M + TILE_M - 1) / TILE_M;
    const int m0 = (blockIdx.x % tiles_m) * TILE_M, n0 = (blockIdx.x / tiles_m) * TILE_N;   // rows first: tiles that share weights run together
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int steps = (K + FK - 1) / FK;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(f32_smem);
    // this thread's 16-byte pieces of a stage: piece tid % 8 of rows tid / 8, tid / 8 + 32, ...
    const int pr = tid >> 3, pc = (tid & 7) * 4;
    auto request = [&](const float* __restrict__ src, int row0, int rows, long long ld, int tile_rows, int offset, int it) {
        const bool k_ok = it * FK + pc < K;            // K is a multiple of 4: a piece lies inside or outside
#pragma unroll
        for (int r = pr; r < tile_rows; r += 32) {
            const bool real = k_ok && row0 + r < rows;
            copy16(base + 4u * ((it % STAGES) * STAGE + (offset + r) * FS + pc), real ? src + (size_t)(row0 + r) * ld + it * FK + pc : src, real);
        }
    };
    if (!ahead) qi::pdl_wait();
    for (int it = 0; it < STAGES - 1 && it < steps; ++it) request(w, n0, N, ldw, TILE_N, TILE_M, it);
    if (ahead) qi::pdl_wait();
    for (int it = 0; it < STAGES - 1; ++it) {           // (the weights above belong to the first group)
        if (it < steps) request(x, m0, M, ldx, TILE_M, 0, it);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int it = 0; it < steps; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();          // this stage has landed, and every thread has left the one that is requested next
        if (it + STAGES - 1 < steps) {
            request(w, n0, N, ldw, TILE_N, TILE_M, it + STAGES - 1);
            request(x, m0, M, ldx, TILE_M, 0, it + STAGES - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* xs = f32_smem + (it % STAGES) * STAGE + ty * FS;
        const float* ws = f32_smem + (it % STAGES) * STAGE + (TILE_M + tx) * FS;
#pragma unroll 2
        for (int k = 0; k < FK; k += 4) {
            float a[TM][4];
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 v = *reinterpret_cast<const float4*>(xs + 16 * i * FS + k);
                a[i][0] = v.x; a[i][1] = v.y; a[i][2] = v.z; a[i][3] = v.w;
            }
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float4 v = *reinterpret_cast<const float4*>(ws + 16 * j * FS + k);
                const float b[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                    for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i][kk], b[kk], acc[i][j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty + 16 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + 16 * j;
            if (n < N) y[(size_t)m * ldy + n] = acc[i][j];
        }
    }
}

template <int TM, int TN>
int launch_f32(const float* x, const float* w, float* y, int M, int N, int K, long long ldx, long long ldw, long long ldy, int batch,
               long long sx, long long sw, long long sy, int ahead, cudaStream_t stream) {
    constexpr int smem = f32_stages(TM, TN) * f32_stage_bytes(TM, TN);
    static bool configured = false;
    if (!configured) {
        if (cudaFuncSetAttribute(gemm_f32_kernel<TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
            return qi::fail("gemm_simt: %d bytes of shared memory were refused", smem);
        configured = true;
    }
    const long long tiles = (long long)((M + 16 * TM - 1) / (16 * TM)) * ((N + 16 * TN - 1) / (16 * TN));
    qi::launch(gemm_f32_kernel<TM, TN>, dim3((unsigned)tiles, 1, batch), dim3(256), smem, stream, x, w, y, M, N, K, ldx, ldw, ldy, sx, sw, sy, ahead);
    return qi::check_launch("gemm_f32");
}

// The tile, of 16 TM x 16 TN for TM in 1..8 and TN in {2, 4, 8}: the one whose fullest SM is done first. A tile of
// K = 4096 takes 45 + 5.6 TM TN us of an SM that has others beside it, and 1.6 times that alone (eight warps do not hide their
// own latency). Fitted to all tiles over 8 to 201 rows at four layer shapes; the choice was the best of them or within 4%.
void f32_tile(int M, int N, int batch, int* best_tm, int* best_tn) {
    static const int tns[3] = {2, 4, 8};
    double best = 1e30;
    for (int tm = 1; tm <= 8; ++tm) {
        if (tm == 5) continue;
        for (int c = 0; c < 3; ++c) {
            const int tn = tns[c];
            const long long tiles = (long long)((M + 16 * tm - 1) / (16 * tm)) * ((N + 16 * tn - 1) / (16 * tn)) * batch;
            const long long an_sm = (tiles + 147) / 148;
            const double cost = (an_sm == 1 ? 1.6 : (double)an_sm) * (45.0 + 5.6 * tm * tn);
            if (cost < best) { best = cost; *best_tm = tm; *best_tn = tn; }
        }
    }
}

bool f32_takes(const void* x, int x_dtype, const void* w, int w_dtype, int y_dtype, int M, int N, int K, long long ldx, long long ldw,
               long long sx, long long sw) {
    return x_dtype == qi::kF32 && w_dtype == qi::kF32 && y_dtype == qi::kF32 && K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && sx % 4 == 0 &&
           sw % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0 && (long long)((M + 15) / 16) * ((N + 31) / 32) < 2147483647LL;
}

int run_f32(const float* x, const float* w, float* y, int M, int N, int K, long long ldx, long long ldw, long long ldy, int batch,
            long long sx, long long sw, long long sy, int ahead, cudaStream_t stream) {
    int tm = 1, tn = 2;
    f32_tile(M, N, batch, &tm, &tn);
    switch (tm * 16 + tn) {
#define QI_F32(TM, TN) case TM * 16 + TN: return launch_f32<TM, TN>(x, w, y, M, N, K, ldx, ldw, ldy, batch, sx, sw, sy, ahead, stream);
#define QI_F32_ROW(TM) QI_F32(TM, 2) QI_F32(TM, 4) QI_F32(TM, 8)
        QI_F32_ROW(1) QI_F32_ROW(2) QI_F32_ROW(3) QI_F32_ROW(4) QI_F32_ROW(6) QI_F32_ROW(7) QI_F32_ROW(8)
#undef QI_F32_ROW
#undef QI_F32
    }
    return qi::fail("gemm_simt: no kernel for a tile of %d x %d", 16 * tm, 16 * tn);
}

}  // namespace

extern "C" int qi_gemm_simt(const void* x, int x_dtype, const void* w, int w_dtype, void* y,
                            int y_dtype, int M, int N, int K, long long ldx, long long ldw,
                            long long ldy, cudaStream_t stream) {
    QI_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_simt: bad sizes M=%d N=%d K=%d", M, N, K);
    QI_REQUIRE(ldx >= K && ldw >= K && ldy >= N, "gemm_simt: a leading dimension is smaller than its row");
    QI_REQUIRE((M + BM - 1) / BM <= 65535, "gemm_simt: M=%d is too large for one launch", M);
    if (M == 0) return 0;
    if (f32_takes(x, x_dtype, w, w_dtype, y_dtype, M, N, K, ldx, ldw, 0, 0))
        return run_f32((const float*)x, (const float*)w, (float*)y, M, N, K, ldx, ldw, ldy, 1, 0, 0, 0, 0, stream);
    QI_DISPATCH_DTYPE(x_dtype, TX, {
        QI_DISPATCH_DTYPE(w_dtype, TW, {
            QI_DISPATCH_DTYPE(y_dtype, TY, {
                return launch<TX, TW, TY>(x, w, y, M, N, K, ldx, ldw, ldy, stream);
            });
        });
    });
    return 0;
}

// y[M, N] = x[M, K] . w[N, K]^T, all float32, rows one after the other, w's first rows read ahead of the stream's order (weights, which no
// kernel in flight writes).
extern "C" int qi_gemm_f32_fma(const float* x, const float* w, float* y, int M, int N, int K, cudaStream_t stream) {
    if (M > 0 && N > 0 && K > 0 && f32_takes(x, qi::kF32, w, qi::kF32, qi::kF32, M, N, K, K, K, 0, 0))
        return run_f32(x, w, y, M, N, K, K, K, N, 1, 0, 0, 0, 1, stream);
    return qi_gemm_simt(x, qi::kF32, w, qi::kF32, y, qi::kF32, M, N, K, K, K, N, stream);
}

// A batch of such products in one launch: product b reads x + b * sx, w + b * sw and writes y + b * sy
// (strides in elements). Per-head projections are this: the heads of one activation row lie side by
// side (sx = the head's width, ldx = the row's), each with a weight matrix of its own.
extern "C" int qi_gemm_simt_batched(const void* x, int x_dtype, const void* w, int w_dtype, void* y,
                                    int y_dtype, int M, int N, int K, long long ldx, long long ldw,
                                    long long ldy, int batch, long long sx, long long sw, long long sy,
                                    cudaStream_t stream) {
    QI_REQUIRE(M >= 0 && N > 0 && K > 0 && batch > 0 && batch <= 65535, "gemm_simt_batched: bad sizes M=%d N=%d K=%d batch=%d", M, N, K, batch);
    QI_REQUIRE(ldx >= K && ldw >= K && ldy >= N, "gemm_simt_batched: a leading dimension is smaller than its row");
    QI_REQUIRE((M + BM - 1) / BM <= 65535, "gemm_simt_batched: M=%d is too large for one launch", M);
    if (M == 0) return 0;
    if (f32_takes(x, x_dtype, w, w_dtype, y_dtype, M, N, K, ldx, ldw, sx, sw))
        return run_f32((const float*)x, (const float*)w, (float*)y, M, N, K, ldx, ldw, ldy, batch, sx, sw, sy, 0, stream);
    QI_DISPATCH_DTYPE(x_dtype, TX, {
        QI_DISPATCH_DTYPE(w_dtype, TW, {
            QI_DISPATCH_DTYPE(y_dtype, TY, {
                return launch<TX, TW, TY>(x, w, y, M, N, K, ldx, ldw, ldy, stream, batch, sx, sw, sy);
            });
        });
    });
    return 0;
}
