// Balanced decomposition of the key switch.
#pragma once
#include "gl.cuh"

namespace luthe {

// GEN = false: the RTL's tie rule; GEN = true: the rule of the reference's
// test-vector generator (TFHE-rs), which takes the digit above the top one as
// 0, so that a top digit equal to B/2 stays positive.  Both give the same
// value mod 2^(BL*L); they differ only in that top digit.
template <int BL, int L, bool GEN>
__device__ __forceinline__ void ks_decomp(u64 v, int *d)
{
    // closest_rep = top BL*L bits + round bit; tie rule of
    // balanced_decomp_unfix_sign_round_bit.py:42-101 / decomp_parallel.sv:73-75,142-150
    constexpr int TOT = BL * L;
    constexpr u32 MASK = (1u << BL) - 1, HALF = 1u << (BL - 1);
    u32 rb = (u32)(v >> (63 - TOT)) & 1u;
    u32 c = (u32)(v >> (64 - TOT)) + rb;  // 0 .. 2^TOT
    u32 last_sign = GEN ? 0u : (((c >> (TOT - 1)) & 1u) && ((c & ((1u << (TOT - 1)) - 1)) || rb));
    u32 carry = 0;
#pragma unroll
    for (int i = 0; i < L; i++) {
        u32 raw = (c >> (BL * i)) & MASK;
        u32 nxt = (i + 1 < L) ? ((c >> (BL * (i + 1))) & MASK) : (last_sign ? MASK : 0u);
        u32 tv = raw + carry;
        bool negd = (tv >> BL) || ((tv & HALF) && ((tv & (HALF - 1)) || (nxt & HALF)));
        d[i] = negd ? (int)tv - (1 << BL) : (int)tv;
        carry = negd ? 1u : 0u;
    }
}

}  // namespace luthe
