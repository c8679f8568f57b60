// Host interface of the tensor-core product of 16-bit activations and quantized weights
// (wq_gemm_sm100.cu), shared by the int4 and int8 entry points.
#pragma once

#include "common.cuh"

namespace b200q {

// What b200q_int4_gemv_ex and b200q_int4_linear_ex take, whichever kernel serves the call.
constexpr int32_t kInt4Flags = B200Q_EXACT_WEIGHTS | B200Q_EARLY_DEPENDENTS | B200Q_SWIGLU_INPUT | B200Q_NO_OVERLAP;

enum WqFormat { kWqInt4 = 0, kWqInt8 = 1 };

struct WqProblem {
    WqFormat format;
    const void* x;        // [rows, in] bf16 | f16
    const void* weight;   // int4: [out, in / 2] u8; int8: [out, in] i8
    const void* scale;    // int4: [out, in / group] of x's type; int8: f32 [out, in / group]
    const uint8_t* zero;  // int4: [out, in / group]
    void* y;              // [rows, out] of x's type
    int64_t rows, in, out, group;  // group: inputs a scale covers
    int32_t dtype;
};

// Whether the kernel takes this problem (at least one row; pointers as the entry points check them).
bool wq_gemm_supports(const WqProblem& p);
// What the launch may do while the kernels before it in the stream still run.
enum class WqStart {
    kStreamOrder,  // nothing: an ordinary launch
    kEarly,        // start, set up its barriers and tensor memory, then wait for them
    kFetchAhead,   // fetch and convert weights too: nothing in flight may be writing those
};
int32_t wq_gemm(const char* who, const WqProblem& p, WqStart start, cudaStream_t stream);

// The time a launch for up to 16 rows is expected to take, by the estimate its tile shape is chosen with.
double wq_gemm_us(const WqProblem& p);

// int4_gemv.cu: the same of the decode kernel that 9 to 16 rows of groups of 128 get; -1 where that is
// another one than the kernel with shared activations.
double rows_kernel_us(const WqProblem& p);

// int4_gemv.cu: of this many rows, how many at the end the decode kernels' passes of 16 (or 64) leave
// to the one- and two-row kernel, whose sums take zero point and scale unrounded.
int64_t int4_unrounded_rows(const WqProblem& p, int32_t flags);

}  // namespace b200q
