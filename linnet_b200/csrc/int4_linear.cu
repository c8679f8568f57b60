// Row-count dispatch of the int4 linear layer, the counterpart of the generated
// `_int4_linear` (src/backend/torch_source.cpp:1553-1570): few rows stream the
// weight once through the decode kernel, many rows go to the tcgen05 dequant-GEMM.
#include "wq_gemm.cuh"

using namespace b200q;

// Up to this many rows the tensor-core product starts early (its fetch of the weights runs ahead of
// the kernel before it, as the decode kernels' does).
static constexpr int64_t kOverlapRows = 64;

// Rows from which the tensor-core product is used.  It takes the same time from 1 to 64 rows; the
// decode kernels' grows with the rows, less so for groups of 128, which they are specialised for.
// Decode kernel / tensor-core product, us a launch in a chain on a B200:
//   groups of 128                 8 rows     9 rows    16 rows    32 rows
//     4096 -> 4096              4.8/10.6  11.4/10.6  11.8/10.7  18.2/11.9
//     4096 -> 28672            23.4/31.2  30.5/31.3  31.4/31.3  59.3/31.2
//     14336 -> 4096            13.6/19.7  26.2/19.7  26.6/19.8  50.9/21.0
//     4096 -> 14336           12.5/17.3  15.2/17.4  15.9/17.4  30.0/17.9
//   other groups                  1 row     3 rows     8 rows    16 rows
//     32, 2048 -> 2048          5.1/7.4   5.4/7.4    6.4/7.5    8.2/7.5
//     32, 4096 -> 4096        12.2/10.6 13.7/11.1  17.7/11.2  22.4/11.3
//     32, 4096 -> 28672       42.9/30.2 49.9/30.3  68.2/30.3 109.7/30.5
//     64, 4096 -> 6144        11.0/11.9 12.7/12.4  17.1/13.6  23.5/13.7
//     64, 4096 -> 14336       22.2/17.5 27.0/17.5  35.8/17.6  56.5/17.7
//     256, 4096 -> 4096         6.1/9.8  7.5/10.3  13.9/10.6  18.6/10.6
//     256, 4096 -> 14336      15.0/17.3 19.7/17.3  30.3/17.3  49.4/17.4
// Over 150 drawn shapes one or two rows with other groups came out either way (0.75 to 1.5 times),
// and 9 to 16 rows with groups of 128 lost up to a third where the product's tiles of 128 columns
// leave its last round mostly empty and K is not split (9557 columns: 75 tiles on 148
// multiprocessors, 26.4/38.8; 11468: 90 tiles, 26.3/33.0): those stay with the decode kernels.
static int64_t gemm_rows(int64_t in, int64_t out, int64_t group) {
    constexpr int64_t kSome = int64_t(12) << 20, kMany = int64_t(32) << 20;  // weights: 3072 x 4096, 8192 x 4096
    const int64_t weights = in * out;
    if (group == 128) {
        const int64_t tiles = (out + 127) / 128, sms = sm_count(), rounds = (tiles + sms - 1) / sms;
        return tiles > sms / 2 && tiles * 10 < rounds * sms * 7 ? 17 : 9;
    }
    if (weights < kSome) return 9;
    if (group <= 64) return weights < kMany ? 4 : 3;
    return weights < kMany ? 7 : 3;
}

extern "C" int32_t b200q_int4_linear_ex(const void* x, const uint8_t* packed, const void* scale,
                                        const uint8_t* zero, void* y, int64_t rows, int64_t in,
                                        int64_t out, int64_t group, int32_t dtype, int32_t flags,
                                        void* stream) {
    if (rows >= gemm_rows(in, out, group) && !(flags & B200Q_SWIGLU_INPUT)) {
        const int32_t ok = check_int4_args("int4_linear", x, packed, scale, zero, y, rows, in, out, group, dtype);
        if (ok != B200Q_OK) return ok;
        B200Q_REQUIRE((flags & ~kInt4Flags) == 0, "int4_linear: unknown flag bits %d", flags);
        WqProblem p{kWqInt4, x, packed, scale, zero, y, rows, in, out, group, dtype};
        const WqStart start = (flags & B200Q_NO_OVERLAP) ? WqStart::kStreamOrder
                              : rows <= kOverlapRows     ? WqStart::kFetchAhead
                                                         : WqStart::kEarly;
        // One or two rows past the passes of the decode kernels stay with the kernel that takes their
        // zero points and scales unrounded: a second launch, and sums with the smaller error.
        const int64_t last = int4_unrounded_rows(p, flags), first = rows - last;
        if (last == 0 || first >= gemm_rows(in, out, group)) {
            p.rows = first;
            if (wq_gemm_supports(p)) {
                const int32_t status = wq_gemm("int4_linear", p, start, static_cast<cudaStream_t>(stream));
                if (status != B200Q_OK || last == 0) return status;
                return b200q_int4_gemv_ex(static_cast<const uint16_t*>(x) + first * in, packed, scale, zero,
                                          static_cast<uint16_t*>(y) + first * out, last, in, out, group, dtype, flags, stream);
            }
        }
    }
    return b200q_int4_gemv_ex(x, packed, scale, zero, y, rows, in, out, group, dtype, flags, stream);
}

extern "C" int32_t b200q_int4_linear(const void* x, const uint8_t* packed, const void* scale,
                                     const uint8_t* zero, void* y, int64_t rows, int64_t in,
                                     int64_t out, int64_t group, int32_t dtype, void* stream) {
    return b200q_int4_linear_ex(x, packed, scale, zero, y, rows, in, out, group, dtype, 0, stream);
}
