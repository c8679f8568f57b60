// Row-count dispatch of the int4 linear layer, the counterpart of the generated
// `_int4_linear` (src/backend/torch_source.cpp:1553-1570): few rows stream the
// weight once through the decode kernels, more go to the tensor-core product.
#include "wq_gemm.cuh"

using namespace b200q;

// Up to this many rows the tensor-core product starts early (its fetch of the weights runs ahead of
// the kernel before it, as the decode kernels' does).
static constexpr int64_t kOverlapRows = 64;

// Rows from which the tensor-core product is used.  It takes the same time from 1 to 64 rows; the
// decode kernels' grows with the rows, less so for groups of 128, which they are specialised for.
// Decode kernel / tensor-core product, us a launch in a chain on a B200:
//   groups of 128                 8 rows     9 rows    16 rows    32 rows
//     4096 -> 4096              5.2/10.6  11.0/10.7  11.2/10.7  20.3/11.8
//     4096 -> 28672            23.8/28.7  31.1/28.8  31.9/28.8  59.9/28.7
//     14336 -> 4096            13.8/18.5  25.4/18.5  25.7/18.5  51.2/19.6
//     4096 -> 14336            12.6/15.9  15.3/15.9  16.0/15.9  29.9/16.2
//   other groups                  1 row     3 rows     8 rows    16 rows
//     32, 2048 -> 2048          5.1/7.1   5.4/7.7    6.4/7.7    8.2/7.8
//     32, 4096 -> 4096        12.2/11.2 13.7/11.6  18.3/11.8  23.2/11.8
//     32, 4096 -> 28672       43.1/30.8 50.1/30.8  68.6/30.9 110.4/30.9
//     64, 4096 -> 6144        11.1/11.4 12.8/11.9  17.5/13.1  23.8/13.2
//     64, 4096 -> 14336       22.5/16.2 27.2/16.2  35.8/16.2  56.7/16.2
//     256, 4096 -> 4096         6.6/9.9  7.6/10.4  14.5/10.5  19.3/10.6
//     256, 4096 -> 14336      15.2/15.8 19.9/15.8  30.5/15.9  49.7/15.9
// Over 150 drawn shapes one or two rows with other groups came out either way (0.75 to 1.5 times).
// 9 to 16 rows with groups of 128 and inputs a multiple of 1024 go by the estimates of both kernels: the
// decode kernel wins where its 14-warp blocks all run at once and the product has no even share for
// the multiprocessors (9 rows 8192 -> 7168: 15.5/20.2, 4096 -> 20000: 23.5/27.6, 4096 -> 14336:
// 15.3/15.9), the product nearly everywhere else (left: 4096 -> 5120, 10.8/12.1, 2048 -> 8192, 8.4/11.0, where
// decode blocks of 7 warps come out just even).  For other inputs a third was lost where the
// product's tiles of 128 columns leave its last round mostly empty and K is not split.
static bool product_takes(const WqProblem& p) {
    constexpr int64_t kSome = int64_t(12) << 20, kMany = int64_t(32) << 20;  // weights: 3072 x 4096, 8192 x 4096
    const int64_t weights = p.in * p.out;
    if (p.group == 128) {
        if (p.rows < 9 || p.rows > 16) return p.rows > 16;
        const double decode = rows_kernel_us(p);
        if (decode >= 0) return decode > 1e6 || wq_gemm_us(p) <= decode;
        const int64_t tiles = (p.out + 127) / 128, sms = sm_count(), rounds = (tiles + sms - 1) / sms;
        return !(tiles > sms / 2 && tiles * 10 < rounds * sms * 7);
    }
    if (weights < kSome) return p.rows >= 9;
    if (p.group <= 64) return p.rows >= (weights < kMany ? 4 : 3);
    return p.rows >= (weights < kMany ? 7 : 3);
}

extern "C" int32_t b200q_int4_linear_ex(const void* x, const uint8_t* packed, const void* scale,
                                        const uint8_t* zero, void* y, int64_t rows, int64_t in,
                                        int64_t out, int64_t group, int32_t dtype, int32_t flags,
                                        void* stream) {
    // (fewer rows: the decode kernels, whatever the shape; their entry has the checks)
    if (rows >= 3 && !(flags & B200Q_SWIGLU_INPUT)) {
        const int32_t ok = check_int4_args("int4_linear", x, packed, scale, zero, y, rows, in, out, group, dtype);
        if (ok != B200Q_OK) return ok;
        B200Q_REQUIRE((flags & ~kInt4Flags) == 0, "int4_linear: unknown flag bits %d", flags);
        WqProblem p{kWqInt4, x, packed, scale, zero, y, rows, in, out, group, dtype};
        const WqStart start = (flags & B200Q_NO_OVERLAP) ? WqStart::kStreamOrder
                              : rows <= kOverlapRows     ? WqStart::kFetchAhead
                                                         : WqStart::kEarly;
        // One or two rows past the passes of the decode kernels stay with the kernel that takes their
        // zero points and scales unrounded: a second launch, and sums with the smaller error.
        const int64_t last = int4_unrounded_rows(p, flags);
        p.rows = rows - last;
        if (product_takes(p) && wq_gemm_supports(p)) {
            const int32_t status = wq_gemm("int4_linear", p, start, static_cast<cudaStream_t>(stream));
            if (status != B200Q_OK || last == 0) return status;
            return b200q_int4_gemv_ex(static_cast<const uint16_t*>(x) + p.rows * in, packed, scale, zero,
                                      static_cast<uint16_t*>(y) + p.rows * out, last, in, out, group, dtype, flags, stream);
        }
    }
    return b200q_int4_gemv_ex(x, packed, scale, zero, y, rows, in, out, group, dtype, flags, stream);
}

extern "C" int32_t b200q_int4_linear(const void* x, const uint8_t* packed, const void* scale,
                                     const uint8_t* zero, void* y, int64_t rows, int64_t in,
                                     int64_t out, int64_t group, int32_t dtype, void* stream) {
    return b200q_int4_linear_ex(x, packed, scale, zero, y, rows, in, out, group, dtype, 0, stream);
}
