// Product of 16-bit activations and quantized weights on the Blackwell tensor cores:
//
//   Y[M, N] = X[M, K] . W[N, K]^T,   W = (q - zero) * scale (int4 groups), q * scale (int8)
//
// Stands in for the reference's many-row routes, which dequantize the whole weight with a Triton
// kernel and call cuBLAS (`_int4_weight` + `F.linear`, src/backend/torch_source.cpp:1519-1566;
// torch/quantized.py:90-105), and for its few-row kernels (torch/kernels.py:212-323, :437-592).
// The weight is dequantized tile by tile inside the product and never written to HBM.
//
// The weight is the A operand and lives in TENSOR MEMORY: a dequantizer thread owns one row of W
// (= one lane), turns 64 of its packed weights into 32 registers of 16-bit pairs in natural order
// and stores them with one tcgen05.st; the activations are the B operand, in shared memory as TMA
// wrote them.  Y comes out transposed (lane = column of Y, tensor-memory column = row of Y).
//   * No shared-memory round trip of dequantized weights: per 16 inputs the products read only
//     nx * 32 B of shared memory, so the wide tiles are not bound by its 128 B a clock.
//   * The instruction is 128 rows of W by nx activations, nx any multiple of 16 to 256: 8 rows or
//     a decode batch cost one pass over the weight, and no work is done for padding to 128 rows.
//
// One persistent block per multiprocessor, 24 warps with fixed roles:
//   warps 0-3   epilogue: tensor memory -> registers -> 16-bit -> Y
//   warp  4, 5  TMA producers of X (128 inputs x nx rows a stage) and W (128 inputs x 128 rows)
//   warp  6, 7  issue tcgen05.mma (7 also allocates tensor memory)
//   warps 8-23  dequantizers: four teams of four warps (a warp may touch the 32 lanes of its
//               quarter only); two teams share an ITEM of 128 inputs x 128 rows, half the inputs each
// A block tile is R * 128 rows of W (R accumulators fed by the same activations: wide tiles halve
// the traffic of X that way) by nx rows of X.  Where the tiles would leave multiprocessors idle a
// cluster of k_splits blocks shares a tile, each a slice of K; their f32 sums meet in distributed
// shared memory, in the order of the slices.  No global scratch, no atomics on results.
// Every wait on an mbarrier is bounded: on expiry the block raises an error flag in global memory,
// stops issuing work, waits for its copies in flight, still releases its tensor memory and returns.
//
// What bounds it: for few rows no unit (ncu, 16 x 14336 -> 4096 and 100 x 4096 -> 28672: integer pipe 38 and
// 49 % busy, issue 50 and 62 %, tensor pipe 5 and 48 %, DRAM under 20 %), but an item's way through its
// roles and the multiprocessors left without a tile; for prompts the tensor pipe (72 % busy at
// 2048 x 4096 -> 28672) and the chip's power.  In a chain of launches on a B200, us, against the kernels
// this one took over from (decode kernels in passes, a bf16-only tensor-core kernel with dequantized
// weights in shared memory):
//   int4 g128 bf16    16 x 14336 -> 4096   25.7 -> 18.5     128 x 4096 -> 28672   47 -> 34
//                   2048 x 4096 -> 28672  383..488 -> 362..418 (power)
//   int4 g32           16 x 4096 -> 28672 110.4 -> 30.9
//   int8               64 x 4096 -> 14336 155.7 -> 19.8     200 x 4096 -> 14336  501.7 -> 27.8
// Slower than the kernel before at two sizes found: 256 x 4096 -> 28672 54 -> 58 and 512 x 4096 -> 14336
// 53 -> 57, where its tiles of 128 columns leave half of a second round of multiprocessors idle.
#include <atomic>

#include "mma.cuh"
#include "umma.cuh"
#include "wq_gemm.cuh"

namespace b200q {
namespace {

constexpr int kTileRows = 128;  // rows of W per accumulator: the lanes of tensor memory
constexpr int kStep = 64;       // inputs a dequantizer thread takes at a time; of a 128-byte swizzled row of X
constexpr int kChunk = 128;     // inputs of an item
constexpr int kXWarp = 4, kWWarp = 5, kMmaWarp = 6, kAllocWarp = 7, kFirstDequantWarp = 8;  // 6 and 7 issue products
constexpr int kThreads = 24 * 32;
constexpr uint32_t kTmemColumns = 512;
constexpr int kSlotColumns = kChunk / 2;  // an item in tensor memory: two 16-bit values a column
constexpr int kMaxXStages = 8, kMaxWStages = 16, kMaxSlots = 4;
constexpr int kMaxShared = 227 * 1024;
constexpr int kAlignment = 1024;  // of the swizzled tiles
constexpr int kMaxSplits = 8;

struct WqArgs {
    const void* scale;
    const uint8_t* zero;
    uint16_t* y;
    int M, K, N;
    int groups;               // scales a row of W
    uint32_t steps_per_group; // 2^32 / (kSteps a scale covers), rounded up; 0: one of them or less
    int m_tiles, tiles;
    int nx;                   // rows of X per tile
    int R;                    // blocks of 128 rows of W per tile
    int issuers;              // accumulators and issuing warps at work: R = 2 has two, R = 1 one or two
    int k_splits;
    int chunks;               // ceil(K / 128)
    int x_stages, w_stages, slots, acc_bufs;
    uint32_t w_ring, exchange, barriers;  // offsets in shared memory (the ring of X is at 0)
    int pairs;                // Y can be written in pairs of columns
    int wait_weights;         // weights may come from the kernel before this one
};

// Non-zero after a bounded wait expired in some launch on this device (the value
// names the waiting role); read back by b200q_int4_gemm_status().
__device__ int g_gemm_error = 0;

using namespace umma;

struct Pipeline {  // shared-memory barriers and the tensor-memory base address
    uint64_t full_x[kMaxXStages], empty_x[kMaxXStages];
    uint64_t full_w[kMaxWStages], empty_w[kMaxWStages];  // empty: one arrival per dequantizer warp of two teams
    uint64_t full_a[kMaxSlots], empty_a[kMaxSlots];      // full: the eight warps of two teams
    uint64_t acc_full[2][2], acc_empty[2][2];  // [buffer][issuer]
    uint64_t sums_full, sums_empty;  // K slices: every epilogue warp of the cluster
    uint32_t tmem_base;
};

// ---- 16-bit weights of one row, natural order -------------------------------------------------

// Eight 4-bit weights -> four pairs, (q - zero) * scale rounded once.  The integer pipe is what
// the dequantizers are bound by, so most of the work is left to the multiply-add pipe: byte i holds
// weights 2i (low bits) and 2i + 1; with the other four bits cleared (two LOP3 a word) a byte in the
// low bits of a 16-bit float reads as q (or 16 q) times the type's smallest subnormal, and one
// multiply-add with kSpread makes q - zero of it, exactly, times 1 / kBack; the scale brings kBack
// with it.  6 integer instructions a word against 9 for (magic + q) - (magic + zero).
template <typename T>
struct Widen4;
template <>
struct Widen4<__nv_bfloat16> {  // smallest subnormal 2^-133
    static constexpr uint32_t kSpread = 0x7D007F00u;  // (2^127, 2^123)
    static constexpr uint32_t kMinus = 0xFF00FF00u;   // -2^127
    static constexpr uint32_t kBack = 0x42804280u;    // 2^6
    static constexpr uint32_t kInfinity = 0x7F80u;
    __device__ static __forceinline__ uint32_t fma(uint32_t a, uint32_t b, uint32_t c) {
        uint32_t r;
        asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
        return r;
    }
    __device__ static __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
        uint32_t r;
        asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
        return r;
    }
};
template <>
struct Widen4<__half> {  // smallest subnormal 2^-24
    static constexpr uint32_t kSpread = 0x68007800u;  // (2^15, 2^11)
    static constexpr uint32_t kMinus = 0xF800F800u;   // -2^15
    static constexpr uint32_t kBack = 0x60006000u;    // 2^9
    static constexpr uint32_t kInfinity = 0x7C00u;
    __device__ static __forceinline__ uint32_t fma(uint32_t a, uint32_t b, uint32_t c) {
        uint32_t r;
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
        return r;
    }
    __device__ static __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
        uint32_t r;
        asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
        return r;
    }
};
// `minus_zero`: -zero / kBack, `scale`: scale * kBack, each twice.
template <typename T>
__device__ __forceinline__ void widen_int4(uint32_t w, uint32_t minus_zero, uint32_t scale, uint32_t* out) {
    using W = Widen4<T>;
    const uint32_t even = w & 0x0F0F0F0Fu, odd = w & 0xF0F0F0F0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        // (even byte i, 0, odd byte i, 0): the zeros are the even byte's sign
        uint32_t spread;
        asm("prmt.b32 %0, %1, %2, %3;" : "=r"(spread) : "r"(even), "r"(odd), "r"(0x8480u + uint32_t(i) * 0x1111u));
        out[i] = W::mul(W::fma(spread, W::kSpread, minus_zero), scale);
    }
}
// The same for scales that kBack would take out of the type's range (or that are not finite).
template <typename T>
__device__ __forceinline__ void widen_int4_huge(uint32_t w, uint32_t zero, uint32_t scale, uint32_t* out) {
    const uint32_t high = w >> 4, bias = Half16<T>::kMagic + zero * 0x00010001u;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        out[i] = sub_mul<T>(lop3_and_or(__byte_perm(w, high, uint32_t(0x4400 + i * 0x1111)), 0x000F000Fu, Half16<T>::kMagic),
                            bias, scale);
}

// Four int8 weights -> two pairs, w * scale in f32 rounded once (the reference's arithmetic,
// `(w.float() * scale).to(dtype)`, torch/quantized.py:193).  w + 128 in the low byte of 2^23 reads as
// 2^23 + 128 + w; two of them an instruction.
template <typename T>
__device__ __forceinline__ void widen_int8(uint32_t w, float scale, uint32_t* out) {
    const uint32_t u = w ^ 0x80808080u;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        uint32_t lo = __byte_perm(u, 0x4B000000u, uint32_t(0x7440 + 2 * i)), hi = __byte_perm(u, 0x4B000000u, uint32_t(0x7441 + 2 * i));
        asm("{\n.reg .b64 v, c;\n"
            "mov.b64 v, {%0, %1};\n"
            "mov.b64 c, {%2, %2};\n"
            "add.rn.f32x2 v, v, c;\n"
            "mov.b64 c, {%3, %3};\n"
            "mul.rn.f32x2 v, v, c;\n"
            "mov.b64 {%0, %1}, v;\n}"
            : "+r"(lo), "+r"(hi)
            : "r"(__float_as_uint(-8388736.0f)), "r"(__float_as_uint(scale)));  // 2^23 + 128
        out[i] = Half16<T>::pack(__uint_as_float(lo), __uint_as_float(hi));
    }
}

// The scales (and zero points) of one item of one row, as loaded.
template <int FORMAT, int GPS>
struct ItemScales {
    uint32_t scale[FORMAT == kWqInt4 ? (GPS + 1) / 2 : GPS];
    uint32_t zero;
};

// `scale`, `zero`: of this row of W; `ks`: which 64 inputs.
template <int FORMAT, int GPS>
__device__ __forceinline__ ItemScales<FORMAT, GPS> load_scales(const void* scale, const uint8_t* zero, uint32_t ks,
                                                               uint32_t steps_per_group) {
    ItemScales<FORMAT, GPS> s = {};
    // (steps_per_group: 2^32 / the number of steps a scale lasts, rounded up; 0 where that is one)
    const uint32_t at = GPS > 1 ? ks * GPS : steps_per_group != 0 ? __umulhi(ks, steps_per_group) : ks;
    if constexpr (FORMAT == kWqInt4) {
        const uint16_t* from = static_cast<const uint16_t*>(scale) + at;
        if constexpr (GPS == 1) {
            s.scale[0] = __ldg(from);
            s.zero = __ldg(zero + at);
        } else if constexpr (GPS == 2) {
            s.scale[0] = __ldg(reinterpret_cast<const uint32_t*>(from));
            s.zero = __ldg(reinterpret_cast<const uint16_t*>(zero + at));
        } else {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(from));
            s.scale[0] = v.x, s.scale[1] = v.y;
            s.zero = __ldg(reinterpret_cast<const uint32_t*>(zero + at));
        }
    } else {
        const uint32_t* from = static_cast<const uint32_t*>(scale) + at;
        if constexpr (GPS == 1) {
            s.scale[0] = __ldg(from);
        } else if constexpr (GPS == 2) {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(from));
            s.scale[0] = v.x, s.scale[1] = v.y;
        } else {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(from));
            s.scale[0] = v.x, s.scale[1] = v.y, s.scale[2] = v.z, s.scale[3] = v.w;
        }
    }
    return s;
}

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}
// 32 columns of this thread's lane.
__device__ __forceinline__ void tmem_store_32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
        "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]),
        "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
// 16 columns of this thread's lane.
__device__ __forceinline__ void tmem_ask_16(uint32_t (&v)[16], uint32_t taddr) {  // v is there after tmem_wait()
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait(uint32_t (&v)[16]) {  // (v passes through: no use of it moves above)
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
                 :
                 : "memory");
}
__device__ __forceinline__ void tmem_load_16(uint32_t (&v)[16], uint32_t taddr) {
    tmem_ask_16(v, taddr);
    tmem_wait(v);
}
// D[tmem] (+)= A[tmem] . B[smem]^T, 128 x N x 16, 16-bit inputs, f32 accumulate.
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void fence_cluster() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }
// The bounded waits of a whole warp: every lane waits (and so sees what the barrier guards), all
// lanes get the same answer.  The second form acquires what other blocks of the cluster released.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, int code) {
    return __all_sync(0xFFFFFFFFu, mbar_wait(bar, parity, &g_gemm_error, code));
}
__device__ __forceinline__ bool warp_wait_cluster(uint64_t* bar, uint32_t parity, int code) {
    return __all_sync(0xFFFFFFFFu, mbar_wait_cluster(bar, parity, &g_gemm_error, code));
}
// A producer that gave up: waits (bounded) for the copies it has in flight, which would otherwise
// land in the shared memory of a block that has left.  `s`, `lap`: where the ring stood.
__device__ __forceinline__ void drain(uint64_t* full, int stages, int s, uint32_t lap) {
    for (int i = 0; i < stages; ++i) {
        if (lap == 0 && i >= s) break;
        mbar_wait(&full[i], (i < s ? lap : lap - 1) & 1, &g_gemm_error, 11);
    }
}

template <typename T, int FORMAT, int GPS>
__global__ void __launch_bounds__(kThreads, 1)
wq_gemm_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const WqArgs a) {
    using H = Half16<T>;
    constexpr int kRowBytes = FORMAT == kWqInt4 ? kChunk / 2 : kChunk;  // of a stage of W
    constexpr uint32_t kWStage = kTileRows * kRowBytes;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + kAlignment - 1) &
                                               ~uintptr_t(kAlignment - 1));
    Pipeline* pipe = reinterpret_cast<Pipeline*>(smem + a.barriers);
    const int warp = __shfl_sync(0xFFFFFFFFu, int(threadIdx.x) / 32, 0), lane = threadIdx.x % 32;
    const int nx = a.nx, R = a.R, issuers = a.issuers, splits = a.k_splits, split = int(blockIdx.x) % splits;
    const int tile_first = int(blockIdx.x) / splits, tile_stride = int(gridDim.x) / splits;
    const int chunk0 = int(int64_t(a.chunks) * split / splits), chunk1 = int(int64_t(a.chunks) * (split + 1) / splits);
    const int span = chunk1 - chunk0;
    const uint32_t x_half = uint32_t(nx) * (kStep * 2), x_stage = 2 * x_half;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.x_stages; ++s) mbar_init(&pipe->full_x[s], 1), mbar_init(&pipe->empty_x[s], uint32_t(R));
        for (int s = 0; s < a.w_stages; ++s) mbar_init(&pipe->full_w[s], 1), mbar_init(&pipe->empty_w[s], 8);
        for (int s = 0; s < a.slots; ++s) mbar_init(&pipe->full_a[s], 8), mbar_init(&pipe->empty_a[s], 1);
        for (int b = 0; b < 4; ++b) mbar_init(&pipe->acc_full[b / 2][b % 2], 1), mbar_init(&pipe->acc_empty[b / 2][b % 2], 4);
        mbar_init(&pipe->sums_full, uint32_t(4 * splits));
        mbar_init(&pipe->sums_empty, uint32_t(4 * splits));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kAllocWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&pipe->tmem_base)),
                     "r"(kTmemColumns)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    if (splits > 1) cluster_sync();  // the others' barriers are ready for remote arrivals
    __syncthreads();
    tc_fence_after();
    pdl_launch_dependents();
    const uint32_t tmem = pipe->tmem_base;
    const uint32_t a_columns = kTmemColumns - uint32_t(a.slots) * kSlotColumns;

    if (warp == kXWarp) {
        if (lane == 0) {
            pdl_wait();  // activations may come from the kernel before this one, y may still be read by it
            int s = 0;
            uint32_t lap = 0;
            bool ok = true;
            for (int tile = tile_first; tile < a.tiles && ok; tile += tile_stride) {
                const int m0 = (tile % a.m_tiles) * nx;
                for (int c = chunk0; c < chunk1 && ok; ++c) {
                    if (lap > 0) ok = mbar_wait(&pipe->empty_x[s], (lap - 1) & 1, &g_gemm_error, 1);
                    if (!ok) break;
                    mbar_expect_tx(&pipe->full_x[s], x_stage);
                    tma_load_2d(smem + s * x_stage, &x_map, c * kChunk, m0, &pipe->full_x[s]);
                    tma_load_2d(smem + s * x_stage + x_half, &x_map, c * kChunk + kStep, m0, &pipe->full_x[s]);
                    if (++s == a.x_stages) s = 0, ++lap;
                }
            }
            if (!ok) drain(pipe->full_x, a.x_stages, s, lap);
        }
    } else if (warp == kWWarp) {
        if (lane == 0) {
            if (a.wait_weights) pdl_wait();
            int s = 0;
            uint32_t lap = 0;
            bool ok = true;
            for (int tile = tile_first; tile < a.tiles && ok; tile += tile_stride) {
                const int n0 = (tile / a.m_tiles) * R * kTileRows;
                for (int c = chunk0; c < chunk1 && ok; ++c) {
                    for (int r = 0; r < R && ok; ++r) {
                        if (lap > 0) ok = mbar_wait(&pipe->empty_w[s], (lap - 1) & 1, &g_gemm_error, 2);
                        if (!ok) break;
                        mbar_expect_tx(&pipe->full_w[s], kWStage);
                        tma_load_2d(smem + a.w_ring + size_t(s) * kWStage, &w_map, c * kRowBytes, n0 + r * kTileRows,
                                    &pipe->full_w[s]);
                        if (++s == a.w_stages) s = 0, ++lap;
                    }
                }
            }
            if (!ok) drain(pipe->full_w, a.w_stages, s, lap);
        }
    } else if (warp >= kMmaWarp && warp < kMmaWarp + issuers) {
        // Two issuing warps, each with an accumulator of its own: issuer 0 takes the even items,
        // issuer 1 the odd ones.  With R = 2 those are the two blocks of rows; with R = 1 they are
        // the even and the odd chunks of K, whose sums the epilogue adds.  (One warp's waits, eight
        // products and commits take about 900 clocks, more than the dequantizers need for an item.)
        // Wide tiles (nx > 192) leave tensor memory for one accumulator and one issuer, whose
        // products take longer than that.  The whole warp runs the loop, one elected lane issues.
        // (With two issuers every ring has an even number of stages, or both use every stage: an
        // issuer that left out a lap of a barrier could not tell its phase from the one after next.)
        // kind::f16 instruction descriptor: f32 accumulator, A and B of one 16-bit type, both
        // K-major, M = 128, N = nx
        constexpr uint32_t kType = H::kDtype == B200Q_BF16 ? 1u : 0u;
        const uint32_t idesc = (1u << 4) | (kType << 7) | (kType << 10) | (uint32_t(nx >> 3) << 17) |
                               (uint32_t(kTileRows >> 4) << 24);
        const int issuer = warp - kMmaWarp, c_step = R == 2 ? 1 : issuers;
        const bool leader = elect_one();
        const uint64_t x_desc = smem_desc(smem_u32(smem));
        const uint32_t half_step = x_half >> 4, stage_step = x_stage >> 4;
        uint32_t t = 0, item0 = 0, x0 = 0;  // tiles, items and stages of X before this tile
        bool ok = true;
        for (int tile = tile_first; tile < a.tiles && ok; tile += tile_stride, ++t) {
            const uint32_t buf = a.acc_bufs == 2 ? (t & 1) : 0, use = a.acc_bufs == 2 ? (t >> 1) : t;
            const int j0 = issuers == 1 ? 0 : int((uint32_t(issuer) - item0) & 1u);  // its first item of the tile
            const int c0 = R == 2 ? 0 : j0;
            const uint32_t first = item0 + uint32_t(j0), x_first = x0 + uint32_t(c0);
            uint32_t slot = first % uint32_t(a.slots), a_phase = (first / uint32_t(a.slots)) & 1;
            int s = int(x_first % uint32_t(a.x_stages));
            uint32_t x_phase = (x_first / uint32_t(a.x_stages)) & 1;
            const uint32_t d = tmem + buf * uint32_t(issuers * nx) + uint32_t(issuer * nx);
            if (use > 0) ok = warp_wait(&pipe->acc_empty[buf][issuer], (use - 1) & 1, 3);
            for (int c = c0; c < span && ok; c += c_step) {
                ok = warp_wait(&pipe->full_x[s], x_phase, 4) && warp_wait(&pipe->full_a[slot], a_phase, 5);
                if (!ok) break;
                tc_fence_after();
                if (leader) {
                    const uint32_t w_at = tmem + a_columns + slot * kSlotColumns;
                    const uint64_t desc = x_desc + uint32_t(s) * stage_step;
#pragma unroll
                    for (int kk = 0; kk < kChunk / 16; ++kk) {
                        if (kk == 4 && 2 * (chunk0 + c) + 1 == a.K / kStep) break;  // the second half is past the end of K
                        umma_f16_ts(d, w_at + kk * 8, desc + (kk < 4 ? uint32_t(2 * kk) : half_step + uint32_t(2 * (kk - 4))),
                                    idesc, kk > 0 ? 1u : uint32_t(c > c0));
                    }
                    umma_commit(&pipe->empty_a[slot]);
                    umma_commit(&pipe->empty_x[s]);
                }
                __syncwarp();
                slot += uint32_t(issuers);
                if (slot >= uint32_t(a.slots)) slot -= uint32_t(a.slots), a_phase ^= 1;
                s += c_step;
                if (s >= a.x_stages) s -= a.x_stages, x_phase ^= 1;
            }
            if (leader && ok) umma_commit(&pipe->acc_full[buf][issuer]);
            __syncwarp();
            item0 += uint32_t(span * R);
            x0 += uint32_t(span);
        }
    } else if (warp >= kFirstDequantWarp) {
        // ---- dequantizers ----
        // Teams 0 and 1 take the two halves of the even items, teams 2 and 3 of the odd ones; an
        // item is a stage of W.
        const int team = (warp - kFirstDequantWarp) / 4, half = team & 1, row = (warp & 3) * 32 + lane;
        const uint32_t lane_base = tmem + (uint32_t(warp & 3) << 21) + a_columns + uint32_t(half) * (kStep / 2);
        const int c_step = R == 2 ? 1 : 2;
        const int ks_real = a.K / kStep;
        if (a.wait_weights) pdl_wait();
        uint32_t item0 = 0;  // items before this tile
        bool ok = true;
        for (int tile = tile_first; tile < a.tiles && ok; tile += tile_stride) {
            const int j0 = int((uint32_t(team >> 1) - item0) & 1u);  // this team's first item of the tile
            const int r = R == 2 ? j0 : 0;
            int c = chunk0 + (R == 2 ? 0 : j0);
            const uint32_t first = item0 + uint32_t(j0);
            int s = int(first % uint32_t(a.w_stages));
            uint32_t phase = (first / uint32_t(a.w_stages)) & 1;
            uint32_t slot = first % uint32_t(a.slots), lap = first / uint32_t(a.slots);
            const int n = min((tile / a.m_tiles * R + r) * kTileRows + row, a.N - 1);
            const void* scale = static_cast<const uint8_t*>(a.scale) + size_t(n) * a.groups * (FORMAT == kWqInt4 ? 2 : 4);
            const uint8_t* zero = a.zero + (FORMAT == kWqInt4 ? size_t(n) * a.groups : 0);
            auto scales_of = [&](int chunk) {  // (the last item may be half past the end of K)
                return load_scales<FORMAT, GPS>(scale, zero, uint32_t(min(2 * chunk + half, ks_real - 1)), a.steps_per_group);
            };
            ItemScales<FORMAT, GPS> next = {}, after = {};
            if (c < chunk1) next = scales_of(c);
            if (c + c_step < chunk1) after = scales_of(c + c_step);
            for (; c < chunk1; c += c_step) {
                const ItemScales<FORMAT, GPS> now = next;
                next = after;
                if (c + 2 * c_step < chunk1) after = scales_of(c + 2 * c_step);
                ok = warp_wait(&pipe->full_w[s], phase, 6);
                if (!ok) break;
                const uint32_t to = lane_base + slot * kSlotColumns;
                const uint32_t at = smem_u32(smem + a.w_ring) + uint32_t(s) * kWStage + uint32_t(row * kRowBytes);
                // All 64 weights are ready in registers before the slot is waited for: the time from a
                // slot's release to its refill is on the products' critical path.
                uint32_t v[32];
                if constexpr (FORMAT == kWqInt4) {
                    constexpr int kGroups = GPS;
                    uint32_t sc[kGroups], back[kGroups], minus_zero[kGroups];
                    bool huge = false;
#pragma unroll
                    for (int g = 0; g < kGroups; ++g) {
                        sc[g] = __byte_perm(now.scale[g / 2], 0u, (g & 1) ? 0x3232u : 0x1010u);
                        back[g] = Widen4<T>::mul(sc[g], Widen4<T>::kBack);
                        const uint32_t z = GPS == 1 ? now.zero : (now.zero >> (8 * g)) & 0xFFu;
                        minus_zero[g] = Widen4<T>::mul(z * 0x00010001u, Widen4<T>::kMinus);
                        huge = huge || (back[g] & 0x7FFFu) >= Widen4<T>::kInfinity;
                    }
                    huge = __any_sync(0xFFFFFFFFu, huge);
                    // 16-byte piece p of row r is at p ^ ((r >> 1) & 3) (64-byte swizzle)
#pragma unroll
                    for (int i = 0; i < 2; ++i) {
                        const uint4 q = lds128(at + (uint32_t((2 * half + i) ^ ((row >> 1) & 3)) << 4));
                        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            const int g = (i * 4 + k) * GPS / 8;
                            widen_int4<T>(w[k], minus_zero[g], back[g], v + 16 * i + 4 * k);
                        }
                        if (huge) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const int g = (i * 4 + k) * GPS / 8;
                                const uint32_t z = GPS == 1 ? now.zero : (now.zero >> (8 * g)) & 0xFFu;
                                widen_int4_huge<T>(w[k], z, sc[g], v + 16 * i + 4 * k);
                            }
                        }
                    }
                } else {
                    // 16-byte piece p of row r is at p ^ (r & 7) (128-byte swizzle)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint4 q = lds128(at + (uint32_t((4 * half + i) ^ (row & 7)) << 4));
                        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            widen_int8<T>(w[k], __uint_as_float(now.scale[(i * 4 + k) * GPS / 16]), v + 8 * i + 2 * k);
                        }
                    }
                }
                if (lap > 0) ok = warp_wait(&pipe->empty_a[slot], (lap - 1) & 1, 7);
                if (!ok) break;
                tc_fence_after();
                tmem_store_32(to, v);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                // (the stage of W is handed back after its last word was USED: an arrival right behind
                // the loads can overtake them while the load unit is busy with scattered scales)
                if (lane == 0) mbar_arrive(&pipe->full_a[slot]), mbar_arrive(&pipe->empty_w[s]);
                s += 2;
                if (s >= a.w_stages) s -= a.w_stages, phase ^= 1;
                slot += 2;
                if (slot >= uint32_t(a.slots)) slot -= uint32_t(a.slots), ++lap;
            }
            item0 += uint32_t(span * R);
        }
    } else if (warp < kXWarp) {
        // ---- epilogue (warp w owns tensor-memory lanes 32w .. 32w+31) ----
        float* exchange = reinterpret_cast<float*>(smem + a.exchange);
        const int cps = (nx + splits - 1) / splits;  // K slices: columns this block adds up
        uint32_t t = 0, item0 = 0;
        bool ok = true;
        for (int tile = tile_first; tile < a.tiles && ok; tile += tile_stride, ++t, item0 += uint32_t(span * R)) {
            const int m0 = (tile % a.m_tiles) * nx, live = min(nx, a.M - m0);
            const uint32_t buf = a.acc_bufs == 2 ? (t & 1) : 0, use = a.acc_bufs == 2 ? (t >> 1) : t;
            const uint32_t lanes = tmem + (uint32_t(warp) << 21) + buf * uint32_t(issuers * nx);
            // R = 1 and two issuers: the first of the sums that exists (a tile of one chunk has only
            // one of them), and whether the other does
            const int first_sum = issuers > R && span == 1 ? int(item0 & 1) : 0;
            const bool both = issuers > R && span > 1;
            if (R == 1) {
                ok = warp_wait(&pipe->acc_full[buf][0], use & 1, 8);
                if (ok && issuers == 2) ok = warp_wait(&pipe->acc_full[buf][1], use & 1, 8);
            }
            if (!ok) break;
            tc_fence_after();
            auto sums = [&](uint32_t (&v)[16], int r, int c0) {  // 16 columns of a finished accumulator
                tmem_load_16(v, lanes + uint32_t((R == 1 ? first_sum : r) * nx + c0));
                if (both) {
                    uint32_t u[16];
                    tmem_load_16(u, lanes + uint32_t(nx + c0));
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(u[j]));
                }
            };
            if (splits == 1) {
                for (int r = 0; r < R; ++r) {
                    if (R == 2) {
                        ok = warp_wait(&pipe->acc_full[buf][r], use & 1, 8);
                        if (!ok) break;
                        tc_fence_after();
                    }
                    const int n = (tile / a.m_tiles * R + r) * kTileRows + warp * 32 + lane;
                    auto store = [&](const uint32_t (&v)[16], int c0) {  // 16 rows of Y, this lane's column
                        uint16_t* dst = a.y + size_t(m0 + c0) * a.N + n;
                        if (a.pairs) {
                            // lanes 2i and 2i+1 trade values, so that each stores a pair of
                            // columns of one row of Y: 4-byte stores, two rows an instruction
                            const int odd = lane & 1;
                            dst += odd ? ptrdiff_t(a.N) - 1 : 0;
#pragma unroll
                            for (int j = 0; j < 16; j += 2) {
                                const uint32_t mine = odd ? v[j + 1] : v[j];
                                const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, odd ? v[j] : v[j + 1], 1);
                                const uint32_t packed = odd ? H::pack(__uint_as_float(other), __uint_as_float(mine))
                                                            : H::pack(__uint_as_float(mine), __uint_as_float(other));
                                if (c0 + j + odd < live && n < a.N) *reinterpret_cast<uint32_t*>(dst) = packed;
                                dst += 2 * size_t(a.N);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (c0 + j < live && n < a.N) dst[size_t(j) * a.N] = H::from_float(__uint_as_float(v[j]));
                        }
                    };
                    if (both) {
#pragma unroll 1
                        for (int c0 = 0; c0 < live; c0 += 16) {
                            uint32_t v[16];
                            sums(v, r, c0);
                            store(v, c0);
                        }
                    } else {
                        // the next 16 columns are on their way while these are stored
                        const uint32_t from = lanes + uint32_t((R == 1 ? first_sum : r) * nx);
                        uint32_t v[16], u[16];
                        tmem_ask_16(v, from);
#pragma unroll 1
                        for (int c0 = 0; c0 < live; c0 += 32) {
                            tmem_wait(v);
                            if (c0 + 16 < live) tmem_ask_16(u, from + uint32_t(c0 + 16));
                            store(v, c0);
                            if (c0 + 16 >= live) break;
                            tmem_wait(u);
                            if (c0 + 32 < live) tmem_ask_16(v, from + uint32_t(c0 + 32));
                            store(u, c0 + 16);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&pipe->acc_empty[buf][r]);
                        if (R == 1) mbar_arrive(&pipe->acc_empty[buf][1]);
                    }
                }
            } else {
                // every block of the cluster adds up cps columns: [slice][column][128 lanes]
                if (t > 0) ok = warp_wait_cluster(&pipe->sums_empty, (t - 1) & 1, 9);
                if (!ok) break;
                const uint32_t mine = smem_u32(exchange) + uint32_t(split * cps * kTileRows + warp * 32 + lane) * 4u;
                int owner = 0, within = 0;
                uint32_t remote = map_to_rank(mine, 0);
#pragma unroll 1
                for (int c0 = 0; c0 < nx; c0 += 16) {
                    if (c0 >= live) break;
                    uint32_t v[16];
                    sums(v, 0, c0);
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(remote + uint32_t(within) * (kTileRows * 4u)),
                                     "r"(v[j])
                                     : "memory");
                        if (++within == cps) within = 0, remote = map_to_rank(mine, min(++owner, splits - 1));
                    }
                }
                tc_fence_before();
                fence_cluster();
                __syncwarp();
                if (lane == 0) mbar_arrive(&pipe->acc_empty[buf][0]), mbar_arrive(&pipe->acc_empty[buf][1]);
                if (lane < splits) arrive_cluster(map_to_rank(smem_u32(&pipe->sums_full), lane));
                ok = warp_wait_cluster(&pipe->sums_full, t & 1, 10);
                if (!ok) break;
                const int n = tile / a.m_tiles * kTileRows + warp * 32 + lane;
                const float* from = exchange + warp * 32 + lane;
                for (int c = 0; c < cps; ++c) {
                    const int col = split * cps + c;
                    if (col >= live) break;
                    float sum = 0.0f;
                    for (int src = 0; src < splits; ++src) sum += from[(src * cps + c) * kTileRows];
                    if (n < a.N) a.y[size_t(m0 + col) * a.N + n] = H::from_float(sum);
                }
                fence_cluster();
                __syncwarp();
                if (lane < splits) arrive_cluster(map_to_rank(smem_u32(&pipe->sums_empty), lane));
            }
        }
    }

    // Every role falls through to here, also after an expired wait.
    tc_fence_before();
    __syncthreads();
    if (warp == kAllocWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemColumns)
                     : "memory");
    }
    if (splits > 1) cluster_sync();  // nobody leaves while another may still write or arrive here
}

// ---- host ---------------------------------------------------------------------------------------

struct WqPlan {
    int nx, R, issuers, splits, m_tiles, n_tiles, acc_bufs, slots, x_stages, w_stages;
    size_t w_ring, exchange, barriers, smem;
};

int w_stage_bytes(WqFormat f) { return kTileRows * (f == kWqInt4 ? kChunk / 2 : kChunk); }

// Shared memory and tensor memory of a tile shape; false where they do not suffice.
bool lay_out(WqPlan& p, WqFormat format) {
    const int columns = p.issuers * p.nx;
    p.acc_bufs = 2 * columns + 2 * kSlotColumns <= int(kTmemColumns) ? 2 : 1;
    const int slots = (int(kTmemColumns) - p.acc_bufs * columns) / kSlotColumns;
    if (slots < 2) return false;
    p.slots = slots >= 4 ? 4 : 2;
    const size_t exchange = p.splits > 1 ? size_t(p.nx + p.splits) * kTileRows * 4 : 0;
    const size_t budget = kMaxShared - kAlignment - sizeof(Pipeline) - exchange;
    const size_t x_stage = size_t(p.nx) * kChunk * 2, w_stage = size_t(w_stage_bytes(format));
    // 64 KB of packed weights in flight hide the HBM latency; few activations leave room for more
    p.w_stages = int((p.nx <= 64 ? 96 * 1024 : 64 * 1024) / w_stage);
    const size_t x_stages = (budget - size_t(p.w_stages) * w_stage) / x_stage;
    p.x_stages = x_stages < size_t(kMaxXStages) ? int(x_stages) : kMaxXStages;
    if (p.issuers > p.R) p.x_stages &= ~1;  // (as are w_stages and slots: the issuers take the stages in turn)
    if (p.x_stages < 2) return false;
    p.w_ring = size_t(p.x_stages) * x_stage;
    p.exchange = p.w_ring + size_t(p.w_stages) * w_stage;
    p.barriers = p.exchange + exchange;
    p.smem = p.barriers + sizeof(Pipeline) + kAlignment;
    return true;
}

typedef void (*WqKernel)(const CUtensorMap, const CUtensorMap, const WqArgs);

template <typename T>
WqKernel pick(WqFormat f, int64_t group) {
    const int gps = group >= kStep ? 1 : int(kStep / group);
    if (f == kWqInt4)
        return gps == 1 ? wq_gemm_kernel<T, kWqInt4, 1> : gps == 2 ? wq_gemm_kernel<T, kWqInt4, 2> : wq_gemm_kernel<T, kWqInt4, 4>;
    return gps == 1 ? wq_gemm_kernel<T, kWqInt8, 1>
                    : gps == 2 ? wq_gemm_kernel<T, kWqInt8, 2> : wq_gemm_kernel<T, kWqInt8, 4>;
}

// Clusters of `splits` blocks (one a multiprocessor) that the device holds at a time.
int resident_clusters(int splits) {
    static std::atomic<int> cached[64][kMaxSplits + 1];
    int device = 0;
    if (splits == 1) return sm_count();
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return sm_count() / splits;
    int count = cached[device][splits].load(std::memory_order_relaxed);
    if (count == 0) {
        const WqKernel kernel = wq_gemm_kernel<__nv_bfloat16, kWqInt4, 1>;
        ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), kMaxShared);
        cudaLaunchConfig_t config = {};
        config.gridDim = dim3(unsigned(splits));
        config.blockDim = dim3(kThreads);
        config.dynamicSmemBytes = kMaxShared;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = unsigned(splits);
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        config.attrs = attr;
        config.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&count, kernel, &config) != cudaSuccess || count <= 0) {
            cudaGetLastError();
            count = sm_count() / splits;
        }
        cached[device][splits].store(count, std::memory_order_relaxed);
    }
    return count;
}

// The tile shape and K split with the least estimated time: rounds of tiles times a tile's clocks, and
// what a launch pays once.  An item (128 inputs x 128 rows of W) takes the products `product` a column
// (`wide` times that where one block of rows is fed from wide tiles of X: shared memory), the
// dequantizers `item` and one issuing warp `issue`.  A tile takes `tile` and `tile_column` a column, with K
// split `split_tile` and `exchange_tile` a column more; one that cannot double-buffer its accumulators
// `column` a column for its epilogue, which the others pay once a launch.  `split`, `exchange`: once a
// launch with K split.
struct PlanClocks {
    double item, issue, product, wide, tile, tile_column, column, split_tile, exchange_tile, split, exchange;
};
// Fitted to the launches of every tile shape at 16 to 2048 rows on five weights.  They serve all but long
// prompts over deep weights; those too with fine groups (several scales an item and row: the dequantizers
// take longer) and odd widths (Y is stored by single columns, and the epilogue is long).
constexpr PlanClocks kFewRows = {766, 1031, 3.5, 1.58, 1200, 0, 48, 3200, 78, 0, 0};
// Fitted to the launches of every tile shape at 100 sizes of more rows (to 2048, 2048 to 14336 inputs, 1024
// to 28672 columns), each shape counting by how near its estimate comes to the least.  Long prompts over
// deep weights take this choice where it is the better one by both estimates together: of 38 drawn or
// listed sizes where the two choices differ, 31 do, 4.6 % faster on average (17 % to 5 % slower; the
// other seven came out 8 % faster to 17 % slower).  2048 x 14336 -> 4096 takes 160 columns and two issuers,
// 196 us; kFewRows alone 240 and one, 208 to 230.  Shorter or shallower, 70 sizes came out either way.
constexpr PlanClocks kManyRows = {580, 1040, 3.43, 1.2, 4000, 0, 18, 4600, 130, 0, 0};
constexpr int64_t kManyFrom = 512, kDeepFrom = 3072;
constexpr double kBoth = 0.98;
// Fitted to the times themselves at 16 to 64 rows: for the choice between this kernel and another.
constexpr PlanClocks kFewRowsTime = {470, 620, 3.2, 1.2, 520, 54, 144, 0, 0, 4870, 95};

double plan_clocks(const WqProblem& q, const WqPlan& p, const PlanClocks& k) {
    const int chunks = int((q.in + kChunk - 1) / kChunk);
    const int64_t tiles = int64_t(p.m_tiles) * p.n_tiles, slots = resident_clusters(p.splits);
    double item = k.product * p.nx * (p.R == 1 && p.nx > 128 ? k.wide : 1.0);
    if (item < k.item) item = k.item;
    if (p.issuers == 1 && item < k.issue) item = k.issue;
    const double epilogue = k.column * p.R * p.nx;
    const double tile = double((chunks + p.splits - 1) / p.splits) * p.R * item + k.tile + k.tile_column * p.nx +
                        (p.splits > 1 ? k.split_tile + k.exchange_tile * p.nx : 0) + (p.acc_bufs == 1 ? epilogue : 0);
    return double((tiles + slots - 1) / slots) * tile + (p.acc_bufs == 2 ? epilogue : 0) +
           (p.splits > 1 ? k.split + k.exchange * p.nx : 0);
}

// The shape with the least estimate, and its clocks; 0 where nothing fits.
double choose_plan(const WqProblem& q, const PlanClocks& k, WqPlan* best) {
    const int chunks = int((q.in + kChunk - 1) / kChunk);
    double best_cost = 0;
    bool found = false;
    const int widest = int(q.rows < 256 ? (q.rows + 15) / 16 * 16 : 256);
    int64_t tried = 0;
    for (int nx = widest < 64 ? widest : 64; nx <= widest; nx += 16) {
        const int64_t m_tiles = (q.rows + nx - 1) / nx;
        if (m_tiles == tried) continue;  // a narrower tile has the same count
        tried = m_tiles;
        for (int shape = 0; shape < 3; ++shape) {
            const int R = shape == 2 ? 2 : 1, issuers = shape == 0 ? 1 : 2;
            if (R == 1 && issuers == 2 && nx > 176) continue;  // no better than one issuer with two accumulators
            const int n_tiles = int((q.out + R * kTileRows - 1) / (R * kTileRows));
            for (int splits = 1; splits <= kMaxSplits; ++splits) {
                if (splits > 1 && (R > 1 || nx > 128 || chunks < 2 * splits)) break;
                WqPlan p = {};
                p.nx = nx, p.R = R, p.issuers = issuers, p.splits = splits, p.m_tiles = int(m_tiles), p.n_tiles = n_tiles;
                if (!lay_out(p, q.format)) continue;
                const double cost = plan_clocks(q, p, k);
                if (!found || cost < best_cost) *best = p, best_cost = cost, found = true;
            }
        }
    }
    return best_cost;
}

}  // namespace

double wq_gemm_us(const WqProblem& q) {
    WqPlan p;
    const double clocks = choose_plan(q, kFewRowsTime, &p);
    return clocks > 0 ? clocks / 1155 - 1.06 : 1e9;  // 300 launches of 9 to 16 rows: 4 % off in the middle, 20 at the 90th percentile
}

bool wq_gemm_supports(const WqProblem& p) {
    const bool fine = p.group == 16 || p.group == 32 || (p.group > 0 && p.group % kStep == 0);
    const int64_t gps = p.group > 0 && p.group < kStep ? kStep / p.group : 1;  // scales are loaded that many at a time
    if (p.rows <= 0 || p.out <= 0 || p.in < kStep || p.in % kStep != 0 || !fine) return false;
    if (p.in >= (int64_t(1) << 22) || p.out >= (int64_t(1) << 28) || p.rows >= (int64_t(1) << 28)) return false;
    if (!aligned(p.x, 16) || !aligned(p.weight, 16) || !aligned(p.y, 2)) return false;
    if (p.format == kWqInt4) return aligned(p.scale, size_t(2 * gps)) && aligned(p.zero, size_t(gps));
    return aligned(p.scale, size_t(4 * gps));
}

int32_t wq_gemm(const char* who, const WqProblem& q, WqStart start, cudaStream_t stream) {
    EncodeTiled encode = encode_tiled();
    if (encode == nullptr) return unavailable("%s: the driver has no cuTensorMapEncodeTiled", who);
    WqPlan p;
    if (choose_plan(q, kFewRows, &p) <= 0) return fail("%s: no tile shape for %lld rows", who, (long long)q.rows);
    const bool pairs = q.out % 2 == 0 && aligned(q.y, 4);
    if (q.rows >= kManyFrom && q.in >= kDeepFrom && q.group >= kStep && pairs) {
        WqPlan other;
        choose_plan(q, kManyRows, &other);
        if (plan_clocks(q, other, kManyRows) * plan_clocks(q, other, kFewRows) <
            kBoth * plan_clocks(q, p, kManyRows) * plan_clocks(q, p, kFewRows))
            p = other;
    }

    const cuuint32_t elem[2] = {1, 1};
    CUtensorMap x_map, w_map;
    const cuuint64_t x_dims[2] = {cuuint64_t(q.in), cuuint64_t(q.rows)}, x_strides[1] = {cuuint64_t(q.in) * 2};
    const cuuint32_t x_box[2] = {cuuint32_t(kStep), cuuint32_t(p.nx)};
    CUresult made = encode(&x_map, q.dtype == B200Q_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                           2, const_cast<void*>(q.x), x_dims, x_strides, x_box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200Q_REQUIRE(made == CUDA_SUCCESS, "%s: cuTensorMapEncodeTiled failed (%d)", who, int(made));
    const bool four = q.format == kWqInt4;
    const cuuint64_t row_bytes = cuuint64_t(four ? q.in / 2 : q.in);
    const cuuint64_t w_dims[2] = {row_bytes, cuuint64_t(q.out)}, w_strides[1] = {row_bytes};
    const cuuint32_t w_box[2] = {cuuint32_t(four ? kChunk / 2 : kChunk), cuuint32_t(kTileRows)};
    made = encode(&w_map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(q.weight), w_dims, w_strides, w_box, elem,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, four ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    B200Q_REQUIRE(made == CUDA_SUCCESS, "%s: cuTensorMapEncodeTiled failed (%d)", who, int(made));

    WqArgs a = {};
    a.scale = q.scale, a.zero = q.zero, a.y = static_cast<uint16_t*>(q.y);
    a.M = int(q.rows), a.K = int(q.in), a.N = int(q.out);
    a.groups = int(q.in / q.group);
    const uint64_t items = q.group >= kStep ? uint64_t(q.group / kStep) : 1;
    a.steps_per_group = items > 1 ? uint32_t(((uint64_t(1) << 32) + items - 1) / items) : 0;
    a.m_tiles = p.m_tiles, a.tiles = p.m_tiles * p.n_tiles;
    a.nx = p.nx, a.R = p.R, a.issuers = p.issuers, a.k_splits = p.splits;
    a.chunks = int((q.in + kChunk - 1) / kChunk);
    a.x_stages = p.x_stages, a.w_stages = p.w_stages, a.slots = p.slots, a.acc_bufs = p.acc_bufs;
    a.w_ring = uint32_t(p.w_ring), a.exchange = uint32_t(p.exchange), a.barriers = uint32_t(p.barriers);
    a.pairs = pairs;
    a.wait_weights = start != WqStart::kFetchAhead;

    const WqKernel kernel = q.dtype == B200Q_BF16 ? pick<__nv_bfloat16>(q.format, q.group) : pick<__half>(q.format, q.group);
    const cudaError_t limit = ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), p.smem);
    if (limit != cudaSuccess) return launch_status(who, limit);
    const int slots = resident_clusters(p.splits);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(unsigned((a.tiles < slots ? a.tiles : slots) * p.splits));
    config.blockDim = dim3(kThreads);
    config.dynamicSmemBytes = p.smem;
    config.stream = stream;
    cudaLaunchAttribute attr[2];
    unsigned attrs = 0;
    if (start != WqStart::kStreamOrder) {
        attr[attrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[attrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (p.splits > 1) {
        attr[attrs].id = cudaLaunchAttributeClusterDimension;
        attr[attrs].val.clusterDim.x = unsigned(p.splits);
        attr[attrs].val.clusterDim.y = attr[attrs].val.clusterDim.z = 1;
        ++attrs;
    }
    config.attrs = attr;
    config.numAttrs = attrs;
    return launch_status(who, cudaLaunchKernelEx(&config, kernel, x_map, w_map, a));
}

// Device address of the bounded-wait flag (also used by the other kernels with bounded waits);
// asked for once per device.
int* gemm_error_word() {
    static int* cached[64] = {nullptr};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return nullptr;
    if (cached[device] == nullptr) {
        void* p = nullptr;
        if (cudaGetSymbolAddress(&p, g_gemm_error) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        cached[device] = static_cast<int*>(p);
    }
    return cached[device];
}

}  // namespace b200q

using namespace b200q;

extern "C" int32_t b200q_int4_gemm(const void* x, const uint8_t* packed, const void* scale,
                                   const uint8_t* zero, void* y, int64_t rows, int64_t in, int64_t out,
                                   int64_t group, int32_t dtype, void* stream) {
    const int32_t ok = check_int4_args("int4_gemm", x, packed, scale, zero, y, rows, in, out, group, dtype);
    if (ok != B200Q_OK || rows == 0) return ok;
    const WqProblem p{kWqInt4, x, packed, scale, zero, y, rows, in, out, group, dtype};
    const int64_t items = group / kStep;
    B200Q_REQUIRE(dtype == B200Q_BF16 && group % kStep == 0 && (items & (items - 1)) == 0 &&
                      out * (in / 2) < (int64_t(1) << 32) && wq_gemm_supports(p),
                  "int4_gemm: needs bf16, inputs a multiple of %d, a group of that many times a power of two, a packed "
                  "weight under 4 GB (got in=%lld group=%lld)", kStep, (long long)in, (long long)group);
    return wq_gemm("int4_gemm", p, WqStart::kEarly, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t b200q_int4_gemm_status(void) {
    int flag = 0;
    const cudaError_t err = cudaMemcpyFromSymbol(&flag, g_gemm_error, sizeof(int));
    if (err != cudaSuccess) return fail("int4_gemm_status: %s", cudaGetErrorString(err));
    if (flag != 0) {
        // Reported once: cleared so that later launches wait their full time again.
        const int zero = 0;
        cudaMemcpyToSymbol(g_gemm_error, &zero, sizeof(int));
        return fail("int4_gemm: a bounded wait expired (role %d)", flag);
    }
    return B200Q_OK;
}
