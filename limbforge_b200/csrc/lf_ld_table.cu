// Width -> launcher table of the block-per-output exact sums.
#include "lf_longdot.cuh"
namespace lfd {
#define LF_LONG_DOT_DECLARE(N) void long_dot_##N(const DotParams&, u32*, cudaStream_t);
LF_LONG_DOT_DECLARE(2) LF_LONG_DOT_DECLARE(3) LF_LONG_DOT_DECLARE(4) LF_LONG_DOT_DECLARE(5) LF_LONG_DOT_DECLARE(6) LF_LONG_DOT_DECLARE(7) LF_LONG_DOT_DECLARE(8) LF_LONG_DOT_DECLARE(9)
LF_LONG_DOT_DECLARE(10) LF_LONG_DOT_DECLARE(11) LF_LONG_DOT_DECLARE(12) LF_LONG_DOT_DECLARE(13) LF_LONG_DOT_DECLARE(14) LF_LONG_DOT_DECLARE(15) LF_LONG_DOT_DECLARE(16) LF_LONG_DOT_DECLARE(17)
LF_LONG_DOT_DECLARE(18) LF_LONG_DOT_DECLARE(19) LF_LONG_DOT_DECLARE(20) LF_LONG_DOT_DECLARE(21) LF_LONG_DOT_DECLARE(22) LF_LONG_DOT_DECLARE(23) LF_LONG_DOT_DECLARE(24) LF_LONG_DOT_DECLARE(25)
LF_LONG_DOT_DECLARE(26) LF_LONG_DOT_DECLARE(27) LF_LONG_DOT_DECLARE(28) LF_LONG_DOT_DECLARE(29) LF_LONG_DOT_DECLARE(30) LF_LONG_DOT_DECLARE(31) LF_LONG_DOT_DECLARE(32)
static const LongDotFn kLongDot[33] = {nullptr, nullptr,
    long_dot_2, long_dot_3, long_dot_4, long_dot_5, long_dot_6, long_dot_7, long_dot_8, long_dot_9, long_dot_10, long_dot_11,
    long_dot_12, long_dot_13, long_dot_14, long_dot_15, long_dot_16, long_dot_17, long_dot_18, long_dot_19, long_dot_20, long_dot_21,
    long_dot_22, long_dot_23, long_dot_24, long_dot_25, long_dot_26, long_dot_27, long_dot_28, long_dot_29, long_dot_30, long_dot_31,
    long_dot_32};
LongDotFn long_dot_launcher(int limbs) { return limbs >= 2 && limbs <= 32 ? kLongDot[limbs] : nullptr; }
}  // namespace lfd
