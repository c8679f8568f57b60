// int8 per-channel decode kernel for one or two activation rows: the structure of the int4
// kernel of int4_gemv_tma.cuh (one block per multiprocessor, the weights brought by the TMA
// unit into a ring of shared-memory stages, a producer thread, consumer warps that never issue
// a weight load).
//
//   y[m, n] = scale[n] * sum_k x[m, k] w[n, k]
//
// A byte u = w + 128 (one XOR per word makes the bytes unsigned) becomes a 16-bit float with one
// byte permute and one multiply-add per pair: in bf16 the byte in the low bits reads as u * 2^-133,
// times 2^127 less 2 is (u - 128) / 64, exact in 8 bits; in f16 0x6400 | u is 1024 + u, less 1152 is
// w.  Five instructions (three of the integer pipe) and one MMA a word of four weights.  Before, a
// byte was taken as two 4-bit planes: seven integer instructions and two MMAs a word, and sums of
// (128 + q) that a correction had to bring back; 18.0 us a launch at 4096 -> 14336 against 16.3,
// two rows at 14336 -> 4096 30.2 against 16.6.
// The per-row scale multiplies the finished sum, as in the kernel this one
// relieves for one and two rows (int8_gemv.cu), and as linnet::gemv8 does
// (python/linnet/src/linnet/torch/kernels.py:336-434).
//
// A k-block is 64 inputs (64 bytes of a row); an item is 16 rows x KB k-blocks, one 3-D TMA
// box landing as [KB][16 rows][64 bytes].  A lane's 16 bytes of a row are its 16 inputs of the
// k-block, so the activations are staged once per block as they are: 32 bytes a lane are the B
// fragments of the four words.
#pragma once

#include <cuda.h>

#include "tma_ring.cuh"

namespace b200q {

// Producer threads (one a warp) of a block.  Sending an item (two barrier tests, the byte count, the
// copy) takes one thread about 450 clocks, and the 16 consumers want one more often than that: one
// -> four producers, us a launch: 4096 -> 14336 16.3 -> 13.8, 4096 -> 28672 28.8 -> 22.9 (5.1 TB/s),
// 14336 -> 4096 16.0 -> 13.7, 4096 -> 6144 7.8 -> 6.9.  (The int4 kernel, whose consumers take
// longer, got 2 to 5 % slower.)  Each producer has its own consumers and its own stages of the ring,
// every `producers`-th of both: a producer that left out a lap of a barrier could not tell its phase
// from the one after next, so their number divides the warps of a tile (and with them every round's
// items) and the stages.
constexpr int kProducers = 4;
inline int tma_producers(int wpt) { return wpt % 4 == 0 ? 4 : wpt % 2 == 0 ? 2 : 1; }

struct Tma8Args {
    const void* x;       // [M, K]
    const float* scale;  // [N]
    void* y;             // [M, N]
    int M, K, N;
    int tiles;           // ceil(N / 16)
    int wpt;             // warps per tile
    int opc;             // items per warp and tile; K == 64 * KB * opc * wpt
    int tpc;             // tiles in work at a time per block = WARPS / wpt
    int stages;          // ring stages of KB KiB
    int overlap;         // launched with programmatic stream serialization
    int early;           // dependents may start as soon as this kernel has started
    int* status;         // device word of expired waits
    int producers;       // threads that send items; wpt and stages are multiples of it
};

struct Tma8Layout {
    uint32_t bars, xs, total;
    uint32_t xrow;  // bytes of one activation row in xs
};
template <int WARPS, int KB>
__host__ __device__ inline Tma8Layout tma8_layout(int M, int K, int stages) {
    Tma8Layout l;
    const int kblocks = K / 64;
    l.bars = uint32_t(stages) * (KB * 1024);
    l.xs = (l.bars + uint32_t(stages + 2 * WARPS) * 8 + 127u) & ~127u;
    l.xrow = uint32_t(kblocks) * 128 + (M > 1 ? 16 : 0);
    l.total = l.xs + uint32_t(M) * l.xrow;
    return l;
}

// Two int8 weights (bytes of u = w + 128 that `selector` picks) as a pair: w in f16, w / 64 in bf16.
__device__ __forceinline__ uint32_t widen8(uint32_t u, bool second, __half) {
    const uint32_t v = __byte_perm(u, 0x64646464u, second ? 0x4342u : 0x4140u), bias = 0x64806480u;  // 1152
    const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&v), *reinterpret_cast<const __half2*>(&bias));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t widen8(uint32_t u, bool second, __nv_bfloat16) {
    const uint32_t v = __byte_perm(u, 0u, second ? 0x4342u : 0x4140u);
    uint32_t r;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(v), "r"(0x7F007F00u), "r"(0xC000C000u));  // 2^127, -2
    return r;
}

template <typename T, int WARPS, int KB>
__global__ void __launch_bounds__((WARPS + kProducers) * 32, 1)
int8_gemv_tma_kernel(const __grid_constant__ CUtensorMap wmap, const Tma8Args a) {
    using H = Half16<T>;
    constexpr int MP = 8;
    constexpr uint32_t kItem = KB * 1024;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const int g = lane / 4, t = lane % 4;
    const int M = a.M, K = a.K, N = a.N;
    const int kblocks = K / 64;
    const int S = a.stages;
    const Tma8Layout lay = tma8_layout<WARPS, KB>(M, K, S);
    const uint32_t smem0 = uint32_t(__cvta_generic_to_shared(smem));
    // empty[s], ready[w], taken[w]: see int4_gemv_tma.cuh
    const uint32_t empty0 = smem0 + lay.bars, ready0 = empty0 + uint32_t(S) * 8, taken0 = ready0 + WARPS * 8;

    const int t0 = int((uint32_t(blockIdx.x) * uint32_t(a.tiles)) / gridDim.x);
    const int t1 = int((uint32_t(blockIdx.x + 1) * uint32_t(a.tiles)) / gridDim.x);
    const int active = a.tpc * a.wpt;
    const int rounds = (t1 - t0 + a.tpc - 1) / a.tpc;

    if (int(threadIdx.x) < S + 2 * WARPS) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty0 + threadIdx.x * 8));
        umma::fence_proxy_async();
    }
    __syncthreads();

    if (warp >= WARPS) {
        // ---- producers: items in the order (round, item of the tile, consumer), every one of
        // them a consumer's in `producers` and with it a stage's ------------------------------------
        const int mine = warp - WARPS, producers = a.producers;
        if (lane != 0 || mine >= producers) return;
        if (a.overlap) pdl_launch_dependents();  // this thread never waits on the previous kernel: weights are constants
        int s = mine;
        uint32_t lap = 0;  // times the ring has been gone round
        bool ok = true;
        int n = 0;         // items each consumer has been sent
        for (int round = 0; round < rounds && ok; ++round) {
            const int tiles_here = min(a.tpc, t1 - t0 - round * a.tpc);  // the last round may be short
            for (int o = 0; o < a.opc && ok; ++o, ++n) {
                int tile = t0 + round * a.tpc, part = mine;
                for (int w = mine; w < tiles_here * a.wpt; w += producers) {
                    const uint32_t empty = empty0 + s * 8, ready = ready0 + w * 8;
                    if (lap > 0) ok = bar_wait<true>(empty, (lap - 1) & 1, a.status, 21);
                    if (ok && n > 0) ok = bar_wait<true>(taken0 + w * 8, (n - 1) & 1, a.status, 23);
                    if (!ok) break;
                    bar_expect(ready, kItem);
                    tma_item(smem0 + uint32_t(s) * kItem, &wmap, tile * 16, (part * a.opc + o) * KB, ready);
                    s += producers;
                    if (s >= S) s -= S, ++lap;
                    part += producers;
                    if (part >= a.wpt) part -= a.wpt, ++tile;
                }
            }
        }
        return;
    }

    // ---- consumers ---------------------------------------------------------------------------
    const bool works = warp < active && t0 + warp / a.wpt < t1;
    const int ts = warp / a.wpt, part = warp % a.wpt;
    const uint32_t xs = smem0 + lay.xs;

    if (a.overlap) {
        if (a.early) pdl_launch_dependents();
        pdl_wait();  // activations may come from the kernel ahead of this one
    }

    // Activations: M * (K / 8) pieces of 16 bytes, as they are.
    {
        const uint4* xg = below_pdl_wait(static_cast<const uint4*>(a.x));
        const int row_pieces = kblocks * 8, pieces = M * row_pieces;
        constexpr int threads = WARPS * 32;
        for (int base = 0; base < pieces; base += 4 * threads) {  // four loads in flight a thread
            uint4 raw[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = base + u * threads + int(threadIdx.x);
                if (e < pieces) raw[u] = ld_mutable(xg + e);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const int e = base + u * threads + int(threadIdx.x);
                const int m = e >= row_pieces ? 1 : 0;  // one or two rows
                if (e < pieces) sts128(xs + uint32_t(m) * lay.xrow + uint32_t(e - m * row_pieces) * 16, raw[u]);
            }
        }
    }
    named_barrier(15, WARPS * 32);  // the consumers only: the producer is on its own way
    if (!works) return;

    // ---- this warp's items --------------------------------------------------------------------
    const float kUnit = H::kDtype == B200Q_BF16 ? 64.0f : 1.0f;  // what widen8 divides a weight by
    uint16_t* y = static_cast<uint16_t*>(a.y);
    const uint32_t wl = uint32_t(g) * 64 + t * 16;  // this lane's bytes of a k-block's row g
    const uint32_t x_lane = xs + uint32_t(min(g, M - 1)) * lay.xrow + t * 32;
    bool ok = true;
    int n = 0;
    int s = warp % S;
    const int s_step = active % S;
    const int last_round = t0 + (rounds - 1) * a.tpc;  // its first tile (a warp's own last tile may be in the round before)
    const int s_last = (min(a.tpc, t1 - last_round) * a.wpt) % S;
    const uint32_t ready = ready0 + warp * 8;
    for (int tile = t0 + ts; tile < t1; tile += a.tpc) {
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        uint32_t stage_addr = 0;
        int s_mine = 0;
        for (int o = 0; o < a.opc; ++o, ++n) {
            const int item = part * a.opc + o;
            s_mine = s;
            s += tile >= last_round ? s_last : s_step;
            if (s >= S) s -= S;
            stage_addr = smem0 + uint32_t(s_mine) * kItem;
            if (ok) ok = bar_wait(ready, uint32_t(n) & 1, a.status, 22);
            __syncwarp();  // every lane has seen the phase
            if (lane == 0) bar_arrive(taken0 + warp * 8);
            const uint32_t wq = stage_addr + wl;
            const uint32_t xq = x_lane + uint32_t(item) * (KB * 128);
#pragma unroll
            for (int j = 0; j < KB; ++j) {
                const uint4 q0 = lds128(wq + j * 1024), q1 = lds128(wq + j * 1024 + 512);
                const uint4 b0 = lds128(xq + j * 128), b1 = lds128(xq + j * 128 + 16);
                const uint32_t w0[4] = {q0.x, q0.y, q0.z, q0.w}, w1[4] = {q1.x, q1.y, q1.z, q1.w};
                const uint32_t b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
                float k[2][4];  // two chains
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t u0 = w0[i] ^ 0x80808080u, u1 = w1[i] ^ 0x80808080u;
                    const uint32_t f[4] = {widen8(u0, false, T{}), widen8(u1, false, T{}),   // rows g, g + 8: first pair
                                           widen8(u0, true, T{}), widen8(u1, true, T{})};    // second pair
                    if (i < 2) mma_first<T>(k[i], f, b[2 * i], b[2 * i + 1]);
                    else H::mma(k[i - 2], f, b[2 * i], b[2 * i + 1]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[e] += k[0][e] + k[1][e];
            }
            if (o + 1 < a.opc) {  // hand the stage back; the tile's last one carries the partial sums first
                __syncwarp();
                if (lane == 0) bar_arrive(empty0 + s_mine * 8);
            }
        }
        const bool last_tile = tile + a.tpc >= t1;
        if (last_tile && a.overlap && !a.early) pdl_launch_dependents();

        // The tile's partial sums meet in the stages its warps have just read; the tile's first
        // warp adds them up, applies the rows' scales, stores y and hands the stages back.
        __syncwarp();
        {
            const uint32_t dst = stage_addr + (g * MP + 2 * t) * 4;
            sts32f(dst, acc[0]);
            sts32f(dst + 4, acc[1]);
            sts32f(dst + 8 * MP * 4, acc[2]);
            sts32f(dst + 8 * MP * 4 + 4, acc[3]);
        }
        umma::fence_proxy_async();  // these writes come before the TMA unit's next ones to the stage
        if (a.wpt > 1) named_barrier(1 + ts, a.wpt * 32);
        else __syncwarp();
        if (part == 0) {
            for (int e = lane; e < 16 * M; e += 32) {
                const int row = e % 16, m = e / 16;
                float sum = 0.0f;
                for (int w = 0; w < a.wpt; ++w) {
                    const int sw = s_mine + w < S ? s_mine + w : s_mine + w - S;
                    sum += lds32f(smem0 + uint32_t(sw) * kItem + (row * MP + m) * 4);
                }
                const int nrow = tile * 16 + row;
                if (nrow < N) y[size_t(m) * N + nrow] = H::from_float(sum * kUnit * __ldg(a.scale + nrow));
            }
            __syncwarp();
            if (lane < a.wpt) bar_arrive(empty0 + (s_mine + lane < S ? s_mine + lane : s_mine + lane - S) * 8);
        }
    }
}

// Launch geometry; false when the kernel does not take the shape.
template <int WARPS, int KB>
inline bool tma8_plan(Tma8Args& a, size_t* smem) {
    if (a.K % (64 * KB) != 0 || a.M > 2 || a.M < 1 || !aligned(a.x, 16)) return false;
    const int runs = a.K / (64 * KB);
    int opc = 1;
    while (runs % opc != 0 || runs / opc > WARPS) ++opc;
    a.opc = opc;
    a.wpt = runs / opc;
    if (a.wpt > 32) return false;
    a.tpc = WARPS / a.wpt;
    if (a.wpt > 1 && a.tpc > 14) a.tpc = 14;
    const Tma8Layout fixed = tma8_layout<WARPS, KB>(a.M, a.K, 0);
    const long budget = 226L * 1024 - long(fixed.total);
    long stages = (budget - 2 * WARPS * 8 - 128) / (KB * 1024 + 8);
    if (stages < 4 || stages <= a.wpt) return false;
    if (stages > 96) stages = 96;
    a.producers = tma_producers(a.wpt);
    if (stages / a.producers * a.producers <= a.wpt) a.producers = 1;
    a.stages = int(stages) / a.producers * a.producers;
    *smem = tma8_layout<WARPS, KB>(a.M, a.K, a.stages).total;
    return true;
}

// The weights [N, K] as 64-byte pieces: (byte of the k-block, row, k-block of the row).
template <int KB>
inline bool tma8_weight_map(CUtensorMap* map, const int8_t* w, int N, int K) {
    const umma::EncodeTiled encode = umma::encode_tiled();
    if (encode == nullptr || !aligned(w, 16)) return false;
    const cuuint64_t dims[3] = {64, cuuint64_t(N), cuuint64_t(K / 64)};
    const cuuint64_t strides[2] = {cuuint64_t(K), 64};
    const cuuint32_t box[3] = {64, 16, KB};
    const cuuint32_t elem[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<int8_t*>(w), dims, strides, box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <typename T, int WARPS, int KB>
int32_t launch_tma8(const Tma8Args& a, const int8_t* w, size_t smem, int sms, cudaStream_t stream) {
    auto kernel = int8_gemv_tma_kernel<T, WARPS, KB>;
    CUtensorMap map;
    if (!tma8_weight_map<KB>(&map, w, a.N, a.K)) return fail("int8_linear: the weight tensor map was refused");
    const cudaError_t attr_err = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), smem);
    if (attr_err != cudaSuccess) {
        cudaGetLastError();
        return fail("int8_linear: %zu bytes of shared memory refused: %s", smem, cudaGetErrorString(attr_err));
    }
    const int grid = a.tiles < sms ? a.tiles : sms;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(unsigned(grid), 1, 1);
    config.blockDim = dim3((WARPS + kProducers) * 32, 1, 1);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attr;
    config.numAttrs = a.overlap ? 1 : 0;
    const cudaError_t err = cudaLaunchKernelEx(&config, kernel, map, a);
    if (err != cudaSuccess) {
        cudaGetLastError();
        return fail("int8_linear: launch failed: %s", cudaGetErrorString(err));
    }
    return B200Q_OK;
}

}  // namespace b200q
