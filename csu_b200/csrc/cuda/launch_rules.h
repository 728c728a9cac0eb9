// launch_rules.h -- which build of the gradients and of the DPLUR sweep a mesh gets, as functions of the mesh and the
// device alone.
#pragma once
#include <math.h>

namespace csu {

// Whether k_grad runs with the register budget of few blocks (SMALL): without the spills its undecided components pay
// for, while the blocks an SM has fit in it. Per RK5 iteration on 148 multiprocessors, without -> with (cells, blocks
// an SM):
//   Euler    3,049 156.5 -> 151.2 us, 13,605 (2.9) 147.2 -> 141.1, 20,186 (4.3) 153.5 -> 166.8
//   laminar  13,605 (2.9) 165.7 -> 157.6, 16,198 (3.4) 184.9 -> 202.6
//   SA       9,120 (1.9) 195.3 -> 191.8, 12,182 (2.6) 198.7 -> 222.0
//   SST      9,120 (1.9) 198.8 -> 194.7, 12,182 (2.6) 203.4 -> 228.2
constexpr bool grad_small(int model, int blocks, int sms)
{
    return blocks <= (model == 0 ? 3 : 2) * sms;
}

// waves of `cells` cells on `sms` multiprocessors that hold `per_sm` of them at a time
constexpr long long sweep_waves(long long cells, int per_sm, int sms)
{
    return (cells + (long long)per_sm * sms - 1) / ((long long)per_sm * sms);
}

// Whether the Euler and laminar sweeps trade registers for more cells in flight (k_sweep's WIDE): 1,152 per
// multiprocessor instead of 640 at the compiler's own count. The build with fewer registers is slower cell by cell (its
// loads are less far ahead), so it has to save waves: half of them with FP64 blocks, a third with FP32 blocks. Per
// iteration with 16 sweeps on 148 multiprocessors, PLAIN -> WIDE, wide / plain waves in brackets:
//   laminar FP32  160,904 cells 310 -> 279 us (1/2), 185,606 341 -> 388 (2/2), 210,136 426 -> 412 (2/3),
//                 295,241 576 -> 521 (2/4), 350,514 818 -> 872 (3/4), 499,477 1,166 -> 1,114 (3/6)
//   Euler FP64    168,100 245 -> 231 (1/2), 186,192 267 -> 324 (2/2), 210,222 339 -> 354 (2/3), 294,848 621 -> 607
//                 (2/4), 380,072 767 -> 832 (3/5), 499,848 1,006 -> 1,005 (3/6), 599,850 1,176 -> 1,232 (4/7)
constexpr bool sweep_wide(int model, bool fp32, long long cells, int sms)
{
    if (model != 0) return false;
    const long long plain = sweep_waves(cells, 640, sms), wide = sweep_waves(cells, 1152, sms);
    return fp32 ? 3 * wide <= 2 * plain : 2 * wide <= plain;
}

// Whether the sweeps after the first gather before they know the flags (k_sweep's EARLY): a shorter chain of loads for
// more registers, which pays while few cells share a multiprocessor. The lines lie between the last size that gained
// and the first that did not, per iteration with 16 sweeps on 148 multiprocessors (cells: PLAIN -> EARLY):
//   Euler FP64    34,810 94.3 -> 90.3 us, 39,728 98.8 -> 101.9
//   laminar FP64  34,810 106.7 -> 102.0, 39,728 117.4 -> 119.9
//   Euler FP32    44,987 99.9 -> 94.5, 49,611 106.7 -> 105.5, 55,402 108.5 -> 108.9
//   laminar FP32  44,987 114.5 -> 108.8, 49,611 122.9 -> 122.4, 55,402 128.6 -> 129.2
//   SA FP64       25,264 124.1 -> 115.2, 30,193 130.4 -> 130.4
//   SA FP32       25,264 114.2 -> 113.5, 34,810 120.5 -> 121.2
constexpr bool sweep_early(int model, bool fp32, long long cells, int sms)
{
    return model < 2 && cells <= (long long)sms * (model == 1 ? 192 : fp32 ? 320 : 256);
}

// The builds of k_sweep.
enum { SWEEP_PLAIN, SWEEP_EARLY, SWEEP_WIDE };

// Meshes that share the autotuner's choice: half octaves of the cell count, apart where the sweep build differs (a
// shape timed on one build is wrong for the other: 360,000 cells Euler FP32 752 us an iteration with the shape of
// 300,000's WIDE sweeps, 670 with its own).
inline int tune_class(int model, bool fp32, long long cells, int sms)
{
    const int build = sweep_early(model, fp32, cells, sms)  ? SWEEP_EARLY
                      : sweep_wide(model, fp32, cells, sms) ? SWEEP_WIDE
                                                            : SWEEP_PLAIN;
    return (int)floor(2.0 * log2((double)cells)) * 4 + build;
}

} // namespace csu
