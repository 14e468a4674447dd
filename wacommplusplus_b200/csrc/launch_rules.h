// Rules of the launches that follow from sizes and options alone: plain C++, for the host.
#pragma once

namespace wb {

constexpr int B200_SMS = 148;

// Two full warps per scheduler: up to here the plain step's records are not sorted, and the reference
// arithmetic keeps its velocity stencil in registers.
constexpr int KEEP_RECORDS = 2 * 4 * B200_SMS * 32;
// All resident at once at launch shape 1 of the FP32 step (12 warps per SM).
constexpr int RESIDENT_RECORDS = 12 * B200_SMS * 32;

// Lanes per warp and threads per block (at most maxThreads) of a launch over `count` items: one warp
// per scheduler of the chip before a warp is filled, as blocks of one size on every SM. Such a launch
// is bound by the latency of its substep chain; fewer lanes per warp meet fewer cell changes and
// lines per load. 1,021 records (random walk) per host interval 0.473 -> 0.428 ms, 16,384 in
// reference arithmetic 0.640 -> 0.564 ms; two warps per scheduler: 0.459 and 0.628 ms. From 18,945
// items on the warps are full.
inline void spread_launch(int count, int maxThreads, int &lanes, int &threads) {
    constexpr long long SMS = B200_SMS, WARPS = 4 * SMS;
    const long long per = (count + WARPS - 1) / WARPS;
    lanes = (int)(per < 1 ? 1 : per > 32 ? 32 : per);
    const long long warps = ((long long)count + lanes - 1) / lanes, even = 32 * ((warps + SMS - 1) / SMS);
    threads = even < maxThreads ? (int)even : maxThreads;
}

// Blocks of `items` work items each that cover `count` (1 to 2^31 - 1).
inline int launch_blocks(int count, long long items) {
    return (int)(((long long)count + items - 1) / items);
}

}  // namespace wb
