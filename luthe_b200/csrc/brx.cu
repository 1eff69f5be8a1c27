// Blind rotation on the tensor cores.
//
// One step multiplies the decomposed digits d (two polynomials, 23-bit) by the
// step's BSK (2 x 2 polynomials over Z_p) mod X^2048 + 1.  With Y = X^32 and
// Y^64 = -1 the product is taken at 64 points y:
//
//   forward   a^(y)_x  = sum_j d_{x+32j} y^j                    (x < 32)
//   product   c^(y)_x' = sum_{x<=x'} a_x b_{x'-x} + y sum_{x>x'} a_x b_{32+x'-x}
//   inverse   c_{x'+32j} = 1/64 sum_y c^(y)_x' y^-j
//
// all mod p and all three as matrix products of bytes with exact 32-bit sums
// (tcgen05 kind::i8): a residue is its 8 bytes, a constant w becomes the 8 x 8
// block whose column i holds the bytes of w 2^(8i) mod p, and the 8
// accumulators of an output, weighted 2^(8s), are folded mod p by about 20
// instructions.  No twiddles and no 64-bit multiplies: the integer pipes,
// which bound the butterfly form (kernels.cu, about 470 instructions per
// coefficient and step), are left with the rotation, the decomposition and
// three folds.
//
// The points are z_m = eta^(4m+1) and their inverses (m < 32, eta^128 = 1,
// eta^2 = 8, i = eta^32 = 2^48), which makes one 32-point matrix serve both
// halves of each transform:
//   forward   at z_m        sum_{j<32} (d_j + i d_{j+32}) z_m^j
//             at 1/z_m  -1/z_m times it: sum_{j<32} (d_{63-j} + i d_{31-j}) z_m^j
//   inverse   E_j = sum_m c^(z_m) z_m^-j,  G_j = sum_m c^(1/z_m) z_m^-j with the
//             z_m^31 it is short of:  c_j = E_j + G_{31-j}, c_{j+32} = i (G_{31-j} - E_j)
// The factors left out of the points 1/z_m, -z_m and z_m^31, are -i together
// and, like the 1/64, part of the BSK.
//
// The BSK block of a point is a Toeplitz matrix (the wrap factor y goes into
// the entries above its diagonal), stored as its 62 distinct 8 x 16-byte core
// matrices: with the K order reversed, neighbouring core matrices of the
// operand overlap in memory (128 bytes apart along N, 256 along K), so a block
// takes 8 KB instead of 64 KB and is read by the MMA as it lies.
//
// A point's product needs 128 ciphertexts as MMA rows, so a step has two
// phases over the whole GPU: first pairs of ciphertexts (inverse transform of
// the last step, accumulate, rotate, decompose, forward transform), then
// product units (tile of 128 ciphertexts, point, column).  CTAs meet through
// counters per tile, not through a barrier.  What they exchange (64 KiB per
// ciphertext and step) and the accumulators stay in L2 up to about 300
// ciphertexts; a launch of 592 writes 18 KB per ciphertext and step of it back
// to memory (ncu, 64 steps: 676 MB, 296 ciphertexts 5 MB).
//
// Reference steps: hw/module/pe_pbs feed_rot.sv:305-307, feed_final.sv:324,
// decomp_balseq_core.sv:135-150, ntt_core_gf64, pp_core,
// mod_switch_to_2powerN, acc_core.sv:8-12, sxt_core.sv:8-14.
#include <cuda.h>

#include "brx.cuh"
#include "tc.cuh"
#include "ntt.cuh"

namespace luthe {
namespace brx {

// ---------------------------------------------------------------- constants

static uint64_t h_mul(uint64_t a, uint64_t b) { return (uint64_t)((unsigned __int128)a * b % gl::P); }

// eta^e: a primitive 128-th root of unity, the 32nd power of the 4096-th root
// of the NTT (psi^64 = 8)
static uint64_t h_eta(int e)
{
    uint64_t eta = 0x984ec5194d005735ull, r = 1;
    for (int i = 0; i < 5; i++) eta = h_mul(eta, eta);
    for (e = ((e % 128) + 128) % 128; e > 0; e--) r = h_mul(r, eta);
    return r;
}

// the eight balanced (signed) bytes of w or w - p, whichever fits
static void balanced_bytes(uint64_t w, int8_t *b)
{
    __int128 x = w > gl::P / 2 ? (__int128)w - gl::P : (__int128)w;
    for (int s = 0; s < 8; s++) {
        b[s] = (int8_t)(uint8_t)(uint64_t)x;
        x = (x - b[s]) >> 8;
    }
    if (x != 0) {  // the other representative
        x = w > gl::P / 2 ? (__int128)w : (__int128)w - gl::P;
        for (int s = 0; s < 8; s++) {
            b[s] = (int8_t)(uint8_t)(uint64_t)x;
            x = (x - b[s]) >> 8;
        }
    }
}

// Byte operands of the two transforms, core matrices of 8 rows (s) x 16 bytes,
// signed bytes (most are 0: eta^e is a power of two or a sum of two):
// forward  rows (m, s), K byte 6 j + b: digit j's byte b, then digit j + 32's : byte s of 2^(8b) z_m^j [i 2^(8(b-3)) z_m^j]
// inverse  rows (j, s), K byte 8 m + i (residue m's byte i)                    : byte s of 2^(8i) z_m^-j
// then the table eta^0 .. eta^127
void build_weights(uint8_t *w)
{
    int8_t b8[8];
    for (int o = 0; o < PH; o++)  // output: m (forward), j (inverse)
        for (int in = 0; in < PH; in++) {
            for (int b = 0; b < 6; b++) {
                balanced_bytes(h_mul(1ull << (8 * (b % 3)), h_eta((4 * o + 1) * in + (b < 3 ? 0 : 32))), b8);
                const int kb = 6 * in + b;
                for (int s = 0; s < 8; s++) w[o * 1536 + (kb / 16) * 128 + s * 16 + kb % 16] = (uint8_t)b8[s];
            }
            for (int i = 0; i < 8; i++) {
                balanced_bytes(h_mul(1ull << (8 * i), h_eta(-(4 * in + 1) * o)), b8);
                const int kb = 8 * in + i;
                for (int s = 0; s < 8; s++) w[WF_BYTES + o * 2048 + (kb / 16) * 128 + s * 16 + kb % 16] = (uint8_t)b8[s];
            }
        }
    for (int e = 0; e < 128; e++) {
        const uint64_t v = h_eta(e);
        for (int i = 0; i < 8; i++) w[WF_BYTES + WI_BYTES + e * 8 + i] = (uint8_t)(v >> (8 * i));
    }
}

// ------------------------------------------------------------- BSK expansion
//
// One CTA per (step, row, column): the polynomial's values at the 64 points
// (times 1/64, and -i at the points 1/z_m), then the 62 core matrices of each
// point's Toeplitz block.  Core c holds the byte blocks of the diagonals c - 31
// (its first 8 bytes per row) and c - 30; a negative diagonal -m is y b_{32-m}.
// Runs once per key.
__global__ void __launch_bounds__(256) expand_kernel(const u64 *__restrict__ std_p, const uint8_t *__restrict__ weights,
                                                     uint8_t *__restrict__ bsk)
{
    __shared__ u64 bk[N], eta[128];  // the polynomial, then its values [point][x]
    __shared__ __align__(16) u64 blk[4][BLOCK_BYTES / 8];
    const size_t i = blockIdx.x >> 2;
    const int q = (blockIdx.x >> 1) & 1, col = blockIdx.x & 1, t = threadIdx.x;
    if (t < 128) eta[t] = reinterpret_cast<const u64 *>(weights + WF_BYTES + WI_BYTES)[t];
    for (int e = t; e < N; e += 256) bk[e] = std_p[((i * 2 + q) * 2 + col) * N + e];
    __syncthreads();
    u64 val[N / 256];
#pragma unroll
    for (int v = 0; v < N / 256; v++) {
        const int e = t + 256 * v, p = e / XN, x = e % XN;
        const u32 g = p < PH ? 4 * p + 1 : 128 - (4 * (p - PH) + 1), extra = p < PH ? 0 : 96;  // -i = eta^96
        u64 s = 0;
        for (u32 j = 0; j < PK; j++) s = gl::add(s, gl::mul(bk[x + XN * j], eta[(g * j + extra) & 127]));
        val[v] = gl::canon(gl::div2k(s, 6));
    }
    __syncthreads();
#pragma unroll
    for (int v = 0; v < N / 256; v++) bk[t + 256 * v] = val[v];
    __syncthreads();
    const int sub = t >> 6, tt = t & 63;  // four points at a time
    for (int p0 = 0; p0 < PK; p0 += 4) {
        const int p = p0 + sub;
        if (tt < 2 * XN - 1) {
            const u32 g = p < PH ? 4 * p + 1 : 128 - (4 * (p - PH) + 1);
            const int d = tt - (XN - 1);
            u64 w = d >= 0 ? bk[p * XN + d] : gl::canon(gl::mul(bk[p * XN + d + XN], eta[g]));
            u64 rows[8];
#pragma unroll
            for (int s = 0; s < 8; s++) rows[s] = 0;
#pragma unroll
            for (int b = 0; b < 8; b++) {
#pragma unroll
                for (int s = 0; s < 8; s++) rows[s] |= ((w >> (8 * s)) & 0xFF) << (8 * b);
                w = gl::canon(gl::shl_abs<8>(w));
            }
#pragma unroll
            for (int s = 0; s < 8; s++) {
                if (tt < CORES) blk[sub][tt * 16 + s * 2] = rows[s];
                if (tt > 0) blk[sub][(tt - 1) * 16 + s * 2 + 1] = rows[s];
            }
        }
        __syncthreads();
        for (int e = t; e < (int)(4 * BLOCK_BYTES / 16); e += 256) {
            const int b = e / (int)(BLOCK_BYTES / 16), r = e % (int)(BLOCK_BYTES / 16);
            reinterpret_cast<ulonglong2 *>(bsk + i * STEP_BYTES + ((size_t)((p0 + b) * 2 + col) * 2 + q) * BLOCK_BYTES)[r] =
                reinterpret_cast<ulonglong2 *>(blk[b])[r];
        }
        __syncthreads();
    }
}

cudaError_t launch_expand(const uint64_t *d_std_p, const Workspace &ws, uint32_t n, cudaStream_t s)
{
    expand_kernel<<<n * 4, 256, 0, s>>>(d_std_p, ws.weights, ws.bsk);
    return cudaGetLastError();
}

// ------------------------------------------------------------------- kernel
//
// Sixteen worker warps do all the integer work; one warp each issues the
// product MMAs and the transform MMAs, makes the copies, and publishes finished
// work.  (Twenty warps: five to a scheduler, 96 registers a thread.)

constexpr int WARPS = 16, WORKERS = 32 * WARPS;
constexpr int W_PMMA = WARPS, W_CMMA = WARPS + 1, W_COPY = WARPS + 2;  // and one that publishes
constexpr int THREADS = 32 * (WARPS + 4);
constexpr int STAGES = 5;                  // ring of product operand atoms
constexpr u32 ATOM = TILE * 128;           // 128 ciphertexts x 128 bytes (16 coefficients)
constexpr u32 SM_WF = 0, SM_WI = WF_BYTES;
constexpr u32 SM_BUF = SM_WI + WI_BYTES;
// first phase: the inverse transform's two operands, then two accumulators; the forward transform's two operands
constexpr u32 SM_OP = SM_BUF, SM_FOP = SM_BUF + 65536;
// second phase: Toeplitz blocks of two units, then the ring; the blocks and the
// ring's first stages lie where the accumulators were, which are free before
// the forward transform is done
constexpr u32 SM_W = SM_BUF, WSLOT = 16384, SM_RING = SM_W + 2 * WSLOT;
constexpr int EARLY = (65536 - 2 * WSLOT) / ATOM;  // such stages
constexpr u32 SM_CTL = SM_BUF + 65536 + 49152;
constexpr u32 SMEM_BYTES = SM_CTL + 256;
static_assert(SM_RING % 1024 == 0 && SM_RING + STAGES * ATOM <= SM_CTL && 2 * BLOCK_BYTES <= WSLOT && SMEM_BYTES <= 232448,
              "layout");

// bound on waits that only depend on this CTA's own MMAs and on the drain of
// copies in flight
constexpr u32 OWN_POLLS = 1u << 26;

struct Ctl {
    u64 full[STAGES], empty[STAGES], wfull[2], wempty[2], dfull[2], dempty[2], opfull, dfree, fop, own[2], drain[2];
    u32 tmem, failed, cts_done, units_done, freed;
};
static_assert(sizeof(Ctl) <= 256, "control block");

// grid-wide progress in global memory, one 128-byte line each: the abort flag,
// then per tile the ciphertext steps and the product units finished so far
constexpr u32 LINE = 32;  // u32
__device__ __forceinline__ u32 *ct_count(u32 *sync, u32 tile) { return sync + LINE * (1 + tile); }
__device__ __forceinline__ u32 *unit_count(u32 *sync, u32 tile) { return sync + LINE * (1 + (u32)TILES + tile); }

__device__ __forceinline__ void give_up(Ctl *ctl, u32 *sync)
{
    *(volatile u32 *)&ctl->failed = 1;
    atomicExch(sync, 1u);
}
// Bounded waits: by the device-wide number of polls (times 32, these polls being
// short) and by about half a minute (counted in 2^10 clocks): CTAs of a launch
// may start late, when other work holds their SMs.  They return false once the
// CTA has given up, so that after a wait ran out anywhere every role runs to its
// end without blocking.
constexpr u32 WAIT_KCLOCKS = 60000000;
struct Patience {
    u32 left = WAIT_KCLOCKS, last = (u32)clock();
    // asked every few polls: has this wait lasted too long, or the CTA given up?
    __device__ __forceinline__ bool over(Ctl *ctl)
    {
        if (*(volatile u32 *)&ctl->failed) return true;
        const u32 now = (u32)clock(), gone = (now - last) >> 10;
        last += gone << 10;
        left -= min(gone, left);
        return left == 0;
    }
};
__device__ __forceinline__ bool wait_bar(u64 *m, u32 parity, u32 polls, Ctl *ctl, u32 *sync)
{
    if (polls && tc::mbar_test(m, parity)) return true;
    Patience patience;
    for (u32 it = 0; it < polls; it++) {
        u32 done;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(tc::smem_u32(m)), "r"(parity)
                     : "memory");
        if (done) return true;
        if ((it & 7) == 7 && patience.over(ctl)) break;
    }
    give_up(ctl, sync);
    return false;
}
__device__ __forceinline__ u32 smem_count(u32 *p)
{
    u32 got;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(got) : "r"(tc::smem_u32(p)) : "memory");
    return got;
}
__device__ __forceinline__ u32 load_acquire(const u32 *p)
{
    u32 got;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(p) : "memory");
    return got;
}
__device__ __forceinline__ u32 load_relaxed(const u32 *p)
{
    u32 got;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(got) : "l"(p) : "memory");
    return got;
}
__device__ __forceinline__ bool wait_smem(u32 *p, u32 want, u32 polls, Ctl *ctl, u32 *sync)
{
    Patience patience;
    for (u32 it = 0; it < polls; it++) {
        if (smem_count(p) >= want) return true;
        if ((it & 15) == 15 && patience.over(ctl)) break;
    }
    give_up(ctl, sync);
    return false;
}
__device__ __forceinline__ void add_smem(u32 *p)
{
    asm volatile("red.release.cta.shared::cta.add.u32 [%0], 1;" ::"r"(tc::smem_u32(p)) : "memory");
}
// everything this CTA finished before counts as done for the grid
__device__ __forceinline__ void publish(u32 *p, u32 count)
{
    asm volatile("fence.proxy.async.global;\n\tfence.acq_rel.gpu;\n\tred.relaxed.gpu.global.add.u32 [%0], %1;" ::"l"(p),
                 "r"(count)
                 : "memory");
}
__device__ __forceinline__ void workers_bar() { asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory"); }

// Balanced digits of eight 64-bit torus words whose upper halves are hi[], base
// 2^BW, one level (gl::decomp_to_p), as 24-bit words of three signed bytes.
// Rounding bit, sign and wrap are one addition: z / 2^(32-BW) is d + 2^(BW-1)
// mod 2^BW, and a zero quotient marks the tie t = B/2 (rare): positive unless
// the rounding bit is set (z below its place) under the RTL's rule.  Adding
// 0x808080 and flipping the top bit of each byte makes the bytes signed.
template <int BW>
__device__ __forceinline__ void digits8(const u32 (&hi)[8], u32 tie_floor, u32 *d)
{
    constexpr u32 RB = 1u << (31 - BW), BIAS = 0x808080u - (1u << (BW - 1));
    bool tie = false;
#pragma unroll
    for (int f = 0; f < 8; f++) {
        const u32 z = hi[f] + (0x80000000u + RB);
        d[f] = ((z >> (32 - BW)) + BIAS) ^ 0x808080u;
        tie |= z < 2 * RB;
    }
    if (__builtin_expect(tie, 0)) {
#pragma unroll
        for (int f = 0; f < 8; f++) {
            const u32 z = hi[f] + (0x80000000u + RB);
            if (z < 2 * RB && z >= tie_floor) d[f] = ((1u << BW) + BIAS) ^ 0x808080u;
        }
    }
}
// four 24-bit words as 12 bytes
__device__ __forceinline__ void pack4(u32 a, u32 b, u32 c, u32 d, u32 *w)
{
    w[0] = __byte_perm(a, b, 0x4210);
    w[1] = __byte_perm(b, c, 0x5421);
    w[2] = __byte_perm(c, d, 0x6542);
}

// one 32-byte store (a full sector per thread)
__device__ __forceinline__ void st_v4(u64 *p, u64 a, u64 b, u64 c, u64 d)
{
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a), "l"(b), "l"(c), "l"(d) : "memory");
}

// What one CTA does, in the order in which every role walks it: step by step
// its couples of ciphertexts, number blockIdx + gridDim m, then its product
// units.  A unit is (tile, point, column); units of neighbouring points come in
// pairs, whose products leave together in full 32-byte sectors.  A last round
// that would leave more than half of the CTAs without a pair hands out single
// units, one to a CTA.
struct Plan {
    u32 couples, pairs, units;
    u32 single;  // pair of the single unit, if units is odd
};
__device__ __forceinline__ Plan make_plan(u32 B)
{
    const u32 b = blockIdx.x, g = gridDim.x, all = (B + 1) / 2, work = (B + TILE - 1) / TILE * PK;
    const u32 base = work / g, rem = work % g;
    Plan p;
    p.couples = all > b ? (all - b + g - 1) / g : 0;
    p.pairs = base + (2 * rem > g && b < rem ? 1 : 0);
    p.units = 2 * p.pairs + (2 * rem <= g && b < 2 * rem ? 1 : 0);
    p.single = base * g + (b >> 1);
    return p;
}
struct Unit {
    u32 tile, p, col;
    bool alone;
};
__device__ __forceinline__ Unit get_unit(const Plan &pl, u32 m)  // m-th unit of this CTA in a step
{
    const bool alone = m >= 2 * pl.pairs;
    const u32 pr = alone ? pl.single : blockIdx.x + (m >> 1) * gridDim.x, h = (alone ? blockIdx.x : m) & 1;
    return Unit{pr / PK, ((pr >> 1) & (PH - 1)) * 2 + h, pr & 1, alone};
}
__device__ __forceinline__ u32 tile_cts(u32 B, u32 tile) { return min((u32)TILE, B - tile * TILE); }

template <int BW>
__global__ void __launch_bounds__(THREADS, 1)
    brx_kernel(const u32 *__restrict__ lwe2N, const u64 *__restrict__ luts, const u32 *__restrict__ lut_id, u32 nlut,
               const uint8_t *__restrict__ weights, const uint8_t *__restrict__ bsk, u64 *__restrict__ ev,
               u64 *__restrict__ prod, u64 *__restrict__ acc_g, u64 *__restrict__ out, u32 B, u32 n,
               u32 *__restrict__ err, u32 mlk, u32 tie_rule, u32 *__restrict__ sync, const unsigned long long *polls_p,
               const __grid_constant__ TensorMap prod_map)
{
    extern __shared__ __align__(1024) uint8_t sm[];
    Ctl *ctl = reinterpret_cast<Ctl *>(sm + SM_CTL);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const u32 smem = tc::smem_u32(sm);
    const u32 polls = (u32)min(min(*polls_p, 1ull << 32) * 32, 0xFFFFFFFFull);

    if (tid == 0) {
        for (int i = 0; i < STAGES; i++) {
            tc::mbar_init(&ctl->full[i], 1);
            tc::mbar_init(&ctl->empty[i], 1);
        }
        for (int i = 0; i < 2; i++) {
            tc::mbar_init(&ctl->wfull[i], 1);
            tc::mbar_init(&ctl->wempty[i], 1);
            tc::mbar_init(&ctl->dfull[i], 1);
            tc::mbar_init(&ctl->dempty[i], WARPS);
            tc::mbar_init(&ctl->own[i], 1);
            tc::mbar_init(&ctl->drain[i], 1);
        }
        tc::mbar_init(&ctl->opfull, 1);
        tc::mbar_init(&ctl->dfree, WARPS);
        tc::mbar_init(&ctl->fop, WARPS);
        ctl->failed = ctl->cts_done = ctl->units_done = ctl->freed = 0;
        tc::fence_mbar_init();
    }
    if (warp == W_PMMA) tc::tmem_alloc_512(&ctl->tmem);
    for (u32 i = tid; i < (WF_BYTES + WI_BYTES) / 16; i += THREADS)
        reinterpret_cast<uint4 *>(sm)[i] = reinterpret_cast<const uint4 *>(weights)[i];
    tc::fence_async_smem();
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const u32 tmem = ctl->tmem;  // columns 0-255 and 256-511: points z_m and 1/z_m; units in turn
    const Plan pl = make_plan(B);
    u32 ring = 0, blocks = 0, gathers = 0;  // atoms, units' blocks and couples' products moved (copy and MMA warps)

    if (warp < WARPS) {
        // ------------------------------------------------------------ workers
        const int r = tid & 127, cq = tid >> 7;  // MMA row (TMEM lane); quarter of the columns
        // row = polynomial (column), pair of coefficients mod 32, ciphertext of the couple, coefficient of the pair: the
        // order in which the products' 64-byte pieces (two ciphertexts) land
        const int q = r >> 6, cl = (r >> 1) & 1, x = ((r & 63) >> 2) * 2 + (r & 1);
        const u32 lane_base = (u32)(r & ~31) << 16;
        const u32 tie_floor = tie_rule == TIE_RTL ? 1u << (31 - BW) : 0u;
        // [2][2][N]: takes the operands' place once they are consumed; the second ciphertext's words are swapped in
        // eights (index ^ 8), so that a warp's 16 words of each lie in different banks
        u64 *accs = reinterpret_cast<u64 *>(sm + SM_OP);
        u64 z[16];  // accumulator at x + 32 j: j = 8 cq + e, then j + 32
        u64 held[8];  // products at the first point of a pair
        u32 own = 0, useq = 0;

        auto arrive = [&](u64 *m) {
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(m);
        };
        auto wait_own = [&](int h) {
            wait_bar(&ctl->own[h], own & 1, OWN_POLLS, ctl, sync);
            __syncwarp();
            tc::fence_after();
        };
        auto acc_of = [&](u32 pair) { return acc_g + (size_t)(2 * pair + cl) * 2 * N + q * N + x + XN * 8 * cq; };
        // One step of a pair of ciphertexts.
        auto step_pair = [&](u32 i, u32 pair) {
            const u32 ct = 2 * pair + cl, ctv = min(ct, B - 1);  // the last pair may be half empty
            u64 *acc = acc_of(pair);
            u64 *as = accs + (cl * 2 + q) * N + (x ^ (cl * 8)) + XN * 8 * cq;
            const u32 a = lwe2N[(size_t)ctv * (n + 1) + i];
            if (i == 0) {
                u32 lid = lut_id[ctv];
                if (lid >= nlut) {  // device-resident ids cannot be checked by the host: flag it, stay in bounds
                    if (q == 0 && x == 0 && cq == 0) atomicOr(err, DEVERR_LUT_ID);
                    lid = 0;
                }
                const u64 *lut = luts + (size_t)lid * 2 * N + q * N + x + XN * 8 * cq;
#pragma unroll
                for (int e = 0; e < 16; e++) z[e] = lut[XN * ((e & 7) + (e >> 3) * PH)];
            } else {
                // (loaded here, under the inverse transform; ahead of it they would cost another stage its registers)
#pragma unroll
                for (int e = 0; e < 16; e++) z[e] = __ldcg(acc + XN * ((e & 7) + (e >> 3) * PH));
                // E_j in columns 8 j, G_{31-j} in columns 256 + 8 (31 - j)
                wait_own(cq >> 1);
                const u32 src_e = tmem + lane_base + cq * 64, src_g = tmem + lane_base + 256 + (24 - 8 * cq) * 8;
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    u32 we[16], wg[16];
                    tc::tmem_ld16(src_e + e * 8, we);
                    tc::tmem_ld16(src_g + (6 - e) * 8, wg);
                    tc::tmem_wait16(we);
                    tc::tmem_wait16(wg);
#pragma unroll
                    for (int f = 0; f < 2; f++) {
                        // pair sums of the bytes: E and G small enough (transform weights mostly 0) to add in 32 bits
                        u32 u[4], v[4], t[4], s[4];
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const u32 te = we[8 * f + 2 * k] + (we[8 * f + 2 * k + 1] << 8);
                            const u32 tg = wg[8 * (1 - f) + 2 * k] + (wg[8 * (1 - f) + 2 * k + 1] << 8);
                            u[k] = te + tg;
                            v[k] = tg - te;
                        }
                        // c_j = sum u_k 2^(16k); c_{j+32} = 2^48 sum v_k 2^(16k) with 2^64 = 2^32 - 1, 2^96 = -1
#pragma unroll
                        for (int k = 0; k < 4; k++) t[k] = u[k] + tc::lift(k);
                        s[0] = tc::lift(0) - v[1] - v[3];
                        s[1] = tc::lift(1) - v[2];
                        s[2] = tc::lift(2) + v[1];
                        s[3] = tc::lift(3) + v[0] + v[2];
                        u64 c0, c1;
                        tc::fold2_lifted(t, s, c0, c1);
                        z[e + f] = gl::add_modsw(z[e + f], c0);
                        z[8 + e + f] = gl::add_modsw(z[8 + e + f], c1);
                    }
                }
                tc::fence_before();
                wait_own(1);  // the operands are consumed: the accumulators may take their place
                own++;
            }
#pragma unroll
            for (int e = 0; e < 16; e++) {
                const int j = (e & 7) + (e >> 3) * PH;
                as[XN * j] = z[e];
                acc[XN * j] = z[e];
            }
            workers_bar();  // accumulators complete in shared memory
            if (i == n) {
                // sample extract of coefficient 0 (many-LUT: m N / mlk) of X^-b ACC: 256 threads a ciphertext
                const u32 g = tid >> 8, t = tid & 255, oc = 2 * pair + g;
                if (oc < B) {
                    const u32 body = lwe2N[(size_t)oc * (n + 1) + n];
                    const u64 *ag = accs + g * 2 * N;
                    for (u32 m = 0; m < mlk; m++) {
                        const u32 b = (body + m * (N / mlk)) & (TWO_N - 1);
                        u64 *o = out + ((size_t)oc * mlk + m) * (N + 1);
#pragma unroll
                        for (int e = 0; e < 8; e++) {
                            const u32 oi = t + 256 * e;
                            const u32 src = ((oi == 0 ? 0u : (u32)N - oi) + b) & (TWO_N - 1);
                            u64 w = ag[(src & (N - 1)) ^ (g * 8)];
                            if (src >= (u32)N) w = 0ull - w;
                            __stcs((unsigned long long *)o + oi, oi == 0 ? w : 0ull - w);
                        }
                        if (t == 0) {
                            const u64 w = ag[N + ((b & (N - 1)) ^ (g * 8))];
                            __stcs((unsigned long long *)o + N, b >= (u32)N ? 0ull - w : w);
                        }
                    }
                }
                tc::fence_async_smem();
                arrive(&ctl->dfree);
                if (lane == 0) add_smem(&ctl->freed);
                return;
            }
            // rotate, subtract, decompose: the digits of 8 pairs (j, j + 32) of this row, twice 48 bytes: in order
            // for the points z_m, in reverse for the points 1/z_m
            {
                const u64 *ap = accs + (cl * 2 + q) * N;
                const u32 src = (x + XN * 8 * cq + TWO_N - a) << 20;  // source index mod 2N in the top 12 bits
                u32 d[16];
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    u32 hi[8];
#pragma unroll
                    for (int f = 0; f < 8; f++) {
                        const u32 p = src + ((u32)(XN * (f + g * PH)) << 20);
                        const u64 m = (u64)(int64_t)((int32_t)p >> 31);  // upper half: negated
                        const u64 rot = ap[((p >> 20) & (N - 1)) ^ (cl * 8)];
                        hi[f] = (u32)(((rot ^ m) - z[8 * g + f] - m) >> 32);
                    }
                    digits8<BW>(hi, tie_floor, d + 8 * g);
                }
                uint8_t *fe = sm + SM_FOP + (cq * 3) * 2048 + r * 16, *ff = sm + SM_FOP + 24576 + ((3 - cq) * 3) * 2048 + r * 16;
                u32 w[12];
#pragma unroll
                for (int k = 0; k < 4; k++) pack4(d[2 * k], d[8 + 2 * k], d[2 * k + 1], d[9 + 2 * k], w + 3 * k);
#pragma unroll
                for (int c = 0; c < 3; c++)
                    *reinterpret_cast<uint4 *>(fe + c * 2048) = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
#pragma unroll
                for (int k = 0; k < 4; k++) pack4(d[15 - 2 * k], d[7 - 2 * k], d[14 - 2 * k], d[6 - 2 * k], w + 3 * k);
#pragma unroll
                for (int c = 0; c < 3; c++)
                    *reinterpret_cast<uint4 *>(ff + c * 2048) = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
            }
            tc::fence_async_smem();
            arrive(&ctl->fop);
            if (lane == 0) add_smem(&ctl->freed);  // the rotation has read accs: the next operands may land there
            // evaluations -> the product's operand: atom (polynomial, 16 coefficients), row = ciphertext,
            // K reversed (slot 31 - x), 128-byte swizzle
            const u32 slot = XN - 1 - x, row = ct & (TILE - 1);
            u64 *o = ev + (size_t)(ct / TILE) * TILE_WORDS + (q * 2 + (slot >> 4)) * (ATOM / 8) + row * 16 +
                     (((slot & 15) >> 1) ^ (row & 7)) * 2 + (slot & 1);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                wait_own(h);
                const u32 src = tmem + lane_base + h * 256 + cq * 64;
                u32 w[2][16];
                tc::tmem_ld16(src, w[0]);
#pragma unroll
                for (int e = 0; e < 8; e += 2) {
                    u32(&cur)[16] = w[(e >> 1) & 1];
                    tc::tmem_wait16(cur);
                    if (e < 6) tc::tmem_ld16(src + (e + 2) * 8, w[(e >> 1) & 1 ^ 1]);
                    else if (h == 1) {
                        tc::fence_before();
                        arrive(&ctl->dfree);  // the next inverse transform may overwrite the accumulators
                    }
                    u64 c0, c1;
                    tc::recombine2_signed(cur, c0, c1);
                    u64 *oo = o + (size_t)(h * PH + cq * 8 + e) * 4 * (ATOM / 8);
                    oo[0] = c0;
                    oo[4 * (ATOM / 8)] = c1;
                }
            }
            own++;
            __syncwarp();
            if (lane == 0) add_smem(&ctl->cts_done);
        };

        // accumulators of a unit -> products in global memory, [tile][pair of points][pair of outputs][ciphertext]
        // of 32 bytes (output, point)
        auto drain = [&](const Unit &u) {
            const u32 d = useq & 1;
            wait_bar(&ctl->dfull[d], (useq >> 1) & 1, polls, ctl, sync);
            __syncwarp();
            useq++;
            tc::fence_after();
            u64 *o = prod + (size_t)u.tile * TILE_WORDS + ((u.p >> 1) * XN + u.col * 16 + cq * 4) * (4 * TILE) + r * 4;
            const bool live = u.tile * TILE + r < B;
            const u32 src = tmem + d * 256 + lane_base + cq * 64;
            u32 w[2][16];
            tc::tmem_ld16(src, w[0]);
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                u32(&cur)[16] = w[(e >> 1) & 1];
                tc::tmem_wait16(cur);
                if (e < 6) tc::tmem_ld16(src + (e + 2) * 8, w[(e >> 1) & 1 ^ 1]);
                else {
                    tc::fence_before();
                    arrive(&ctl->dempty[d]);
                }
                u64 c0, c1;
                tc::recombine2_wide(cur, c0, c1);
                u64 *oo = o + (e >> 1) * (4 * TILE);
                if (u.alone) {
                    if (live) {
                        oo[u.p & 1] = c0;
                        oo[2 + (u.p & 1)] = c1;
                    }
                } else if (!(u.p & 1)) {
                    held[e] = c0;
                    held[e + 1] = c1;
                } else if (live) {
                    st_v4(oo, held[e], c0, held[e + 1], c1);
                }
            }
            __syncwarp();
            if (lane == 0) add_smem(&ctl->units_done);
        };

        for (u32 i = 0; i <= n; i++) {
            for (u32 m = 0; m < pl.couples; m++) {
                step_pair(i, blockIdx.x + m * gridDim.x);
            }
            for (u32 m = 0; m < pl.units && i < n; m++) drain(get_unit(pl, m));
        }
    } else if (warp == W_PMMA) {
        // ------------------------------------- product MMAs: D = atoms x Toeplitz blocks
        // (the next atom's barrier is polled before this one's MMAs are issued, which block while the tensor
        // pipe's queue is full: a poll after them would leave the pipe idle)
        if (lane == 0) {
            const u64 da = tc::desc_sw128(smem + SM_RING), dw = tc::desc_plain(smem + SM_W, 256, 128);
            bool good = true, ready = false;
            for (u32 i = 0; i < n && good; i++)
                for (u32 m = 0; m < pl.units && good; m++) {
                    const u32 d = blocks & 1, dt = tmem + d * 256;
                    // the forward transforms' accumulators lie where the units' go
                    if (m == 0) good = wait_smem(&ctl->cts_done, WARPS * pl.couples * (i + 1), polls, ctl, sync);
                    if (blocks >= 2) good = good && wait_bar(&ctl->dempty[d], ((blocks >> 1) - 1) & 1, polls, ctl, sync);
                    good = good && wait_bar(&ctl->wfull[d], (blocks >> 1) & 1, polls, ctl, sync);
                    const u64 wd0 = tc::desc_at(dw, d * WSLOT);
#pragma unroll
                    for (u32 a = 0; a < 4; a++) {
                        const u32 st = ring % STAGES, nx = (ring + 1) % STAGES;
                        if (!ready) good = good && wait_bar(&ctl->full[st], (ring / STAGES) & 1, polls, ctl, sync);
                        if (!good) break;
                        ready = tc::mbar_test(&ctl->full[nx], ((ring + 1) / STAGES) & 1);
                        tc::fence_after();
                        const u64 ad = tc::desc_at(da, st * ATOM);
#pragma unroll
                        for (int s = 0; s < 4; s++)
                            tc::mma_i8(dt, tc::desc_at(ad, s * 32),
                                       tc::desc_at(wd0, (a >> 1) * (u32)BLOCK_BYTES + (a & 1) * 2048 + s * 512),
                                       tc::idesc_i8(256, false, false), s > 0 || a > 0);
                        tc::commit(&ctl->empty[st]);
                        if (a == 3) {
                            tc::commit(&ctl->wempty[d]);
                            tc::commit(&ctl->dfull[d]);
                        }
                        ring++;
                    }
                    blocks++;
                }
        }
        __syncwarp();
    } else if (warp == W_CMMA) {
        // ------------------------------------------------- transform MMAs of each pair
        u32 ops = 0, fops = 0, seq = 0;
        bool good = true;
        for (u32 i = 0; i <= n && good; i++)
            for (u32 m = 0; m < pl.couples && good; m++, seq++) {
                if (seq > 0) good = wait_bar(&ctl->dfree, (seq - 1) & 1, polls, ctl, sync);
                if (i > 0) {
                    good = good && wait_bar(&ctl->opfull, ops & 1, polls, ctl, sync);
                    good = __all_sync(0xFFFFFFFFu, good);
                    if (!good) break;
                    ops++;
                    tc::fence_after();
                    if (lane == 0) {
                        // first the columns of E_j, j < 16, and G_t, t >= 16, which meet in the workers' first half
#pragma unroll
                        for (int h = 0; h < 2; h++) {
#pragma unroll
                            for (int g = 0; g < 2; g++) {
                                const u32 half = g ? 1 - h : h;
#pragma unroll
                                for (int s = 0; s < 8; s++)
                                    tc::mma_i8(tmem + g * 256 + half * 128, tc::desc_plain(smem + SM_OP + g * 32768 + s * 4096, 2048, 128),
                                               tc::desc_plain(smem + SM_WI + half * 16 * 2048 + s * 256, 128, 2048),
                                               tc::idesc_i8(128, false, true), s > 0);
                            }
                            tc::commit(&ctl->own[h]);
                        }
                    }
                    __syncwarp();
                }
                if (i < n) {
                    good = good && wait_bar(&ctl->fop, fops & 1, polls, ctl, sync);
                    good = __all_sync(0xFFFFFFFFu, good);
                    if (!good) break;
                    fops++;
                    tc::fence_after();
                    if (lane == 0) {
#pragma unroll
                        for (int h = 0; h < 2; h++) {
#pragma unroll
                            for (int s = 0; s < 6; s++)
                                tc::mma_i8(tmem + h * 256, tc::desc_plain(smem + SM_FOP + h * 24576 + s * 4096, 2048, 128),
                                           tc::desc_plain(smem + SM_WF + s * 256, 128, 1536), tc::idesc_i8(256, true, true),
                                           s > 0);
                            tc::commit(&ctl->own[h]);
                        }
                    }
                    __syncwarp();
                }
            }
    } else if (warp == W_COPY) {
        // ------------------------------------------------- copies: a couple's products to the inverse transform
        // once its tile's units are done, then the units' operands once their tile is complete
        bool good = true;
        const u32 tiles = (B + TILE - 1) / TILE;
        u32 seq = 0;  // couples so far
        // each lane watches one tile's counter; false if that wait ran out.  The barrier orders what the watching lane
        // acquired before the copies that lane 0 issues: the vote orders no memory.  (Ahead of the vote it costs
        // nothing; after the loop 408 ciphertexts took 1 % longer.)
        auto wait_tile = [&](u32 tile, u32 &complete, bool units, u32 i) {
            Patience patience;
            for (u32 it = 0; !(complete >> tile & 1); it++) {
                const u32 t = min((u32)lane, tiles - 1);
                const u32 got = load_acquire(units ? unit_count(sync, t) : ct_count(sync, t));
                __syncwarp();
                complete = __ballot_sync(0xFFFFFFFFu, got >= (units ? PK * 2 * i : tile_cts(B, t) * (i + 1)));
                const bool over = it >= polls || ((it & 15) == 15 && (patience.over(ctl) || load_relaxed(sync)));
                if (__any_sync(0xFFFFFFFFu, over) && !(complete >> tile & 1)) {
                    give_up(ctl, sync);
                    return false;
                }
            }
            return true;
        };
        for (u32 i = 0; i <= n && good; i++) {
            u32 complete = 0;
            for (u32 m = 0; m < pl.couples && good; m++, seq++) {
                if (i == 0) continue;
                const u32 ct = 2 * (blockIdx.x + m * gridDim.x);
                // this CTA's units are drained (their operands lay here), the last couple's accumulators read
                if (m == 0) good = wait_smem(&ctl->units_done, WARPS * pl.units * i, polls, ctl, sync);
                good = good && wait_smem(&ctl->freed, WARPS * seq, polls, ctl, sync);
                good = __all_sync(0xFFFFFFFFu, good) && wait_tile(ct / TILE, complete, true, i);
                if (good && lane == 0) {
                    tc::fence_async_global();
                    tc::mbar_expect_tx(&ctl->opfull, 65536);
                    // each lands as [pair of points][column, pair of x][ciphertext][x][2]
                    tc::tensor_g2s(sm + SM_OP, &prod_map, (ct & (TILE - 1)) / 2, ct / TILE * PH, &ctl->opfull);
                    tc::tensor_g2s(sm + SM_OP + 32768, &prod_map, (ct & (TILE - 1)) / 2, ct / TILE * PH + PH / 2, &ctl->opfull);
                    gathers++;
                }
            }
            if (i == n || !pl.units || !good) continue;
            good = __all_sync(0xFFFFFFFFu, wait_smem(&ctl->freed, WARPS * seq, polls, ctl, sync));
            complete = 0;
            u32 first = 0;  // atoms of this step
            for (u32 m = 0; m < pl.units && good; m++) {
                const Unit u = get_unit(pl, m);
                const u32 slot = blocks & 1;
                if (blocks >= 2) good = wait_bar(&ctl->wempty[slot], ((blocks >> 1) - 1) & 1, polls, ctl, sync);
                good = __all_sync(0xFFFFFFFFu, good);
                if (!good) break;
                if (lane == 0) {
                    tc::mbar_expect_tx(&ctl->wfull[slot], 2 * BLOCK_BYTES);
                    tc::bulk_g2s(sm + SM_W + slot * WSLOT, bsk + i * STEP_BYTES + (size_t)(u.p * 2 + u.col) * 2 * BLOCK_BYTES,
                                 2 * BLOCK_BYTES, &ctl->wfull[slot]);
                }
                blocks++;
                good = wait_tile(u.tile, complete, false, i);
                if (lane == 0) {
                    tc::fence_async_global();
                    const u64 *src = ev + (size_t)u.tile * TILE_WORDS + (size_t)u.p * 4 * (ATOM / 8);
                    for (u32 a = 0; a < 4 && good; a++, first++) {
                        const u32 st = ring % STAGES;
                        // a stage where the digits lay waits for the forward transforms, as does one of the last step
                        if (first < (u32)STAGES && st >= (u32)EARLY)
                            good = wait_smem(&ctl->cts_done, WARPS * seq, polls, ctl, sync);
                        if (good && ring >= STAGES) good = wait_bar(&ctl->empty[st], (ring / STAGES - 1) & 1, polls, ctl, sync);
                        if (!good) break;
                        tc::mbar_expect_tx(&ctl->full[st], ATOM);
                        tc::bulk_g2s(sm + SM_RING + st * ATOM, src + a * (ATOM / 8), ATOM, &ctl->full[st]);
                        ring++;
                    }
                }
                good = __all_sync(0xFFFFFFFFu, good);
            }
        }
    } else {
        // ------------------------------------------------- publish finished couples and units, in the workers' order
        if (lane == 0) {
            u32 cts = 0, units = 0;
            bool good = true;
            for (u32 i = 0; i < n && good; i++) {
                for (u32 m = 0; m < pl.couples && good; m++) {
                    const u32 ct = 2 * (blockIdx.x + m * gridDim.x);
                    good = wait_smem(&ctl->cts_done, WARPS * ++cts, polls, ctl, sync);
                    if (good) publish(ct_count(sync, ct / TILE), min(2u, B - ct));
                }
                for (u32 m = 0; m < pl.units && good; m++) {
                    const Unit u = get_unit(pl, m);
                    good = wait_smem(&ctl->units_done, WARPS * ++units, polls, ctl, sync);
                    // the products of a pair of points leave with its second unit
                    if (good && (u.alone || (u.p & 1))) publish(unit_count(sync, u.tile), u.alone ? 1 : 2);
                }
            }
        }
    }

    // nothing may still land in this CTA's shared memory or run on its
    // operands when it ends: after a wait that ran out, each issuing thread
    // waits (bounded) for its own MMAs or copies
    __syncwarp();
    __syncthreads();
    if (ctl->failed) {
        bool drained = true;
        if (tid == W_PMMA * 32 || tid == W_CMMA * 32) {
            const int k = warp - W_PMMA;
            tc::commit(&ctl->drain[k]);
            drained = tc::mbar_wait(&ctl->drain[k], 0, OWN_POLLS);
        } else if (tid == W_COPY * 32) {
            for (u32 s = 0; s < STAGES; s++)
                if (ring > s) drained &= tc::mbar_wait(&ctl->full[s], ((ring - 1 - s) / STAGES) & 1, OWN_POLLS);
            for (u32 s = 0; s < 2; s++)
                if (blocks > s) drained &= tc::mbar_wait(&ctl->wfull[s], ((blocks - 1 - s) >> 1) & 1, OWN_POLLS);
            if (gathers) drained &= tc::mbar_wait(&ctl->opfull, (gathers - 1) & 1, OWN_POLLS);
        }
        if (tid == 0) atomicOr(err, DEVERR_TIMEOUT);
        if (!drained) atomicOr(err, DEVERR_DRAIN);
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    __syncwarp();
    if (warp == W_PMMA) tc::tmem_free_512(tmem);
}

cudaError_t set_attributes()
{
    cudaError_t e = cudaFuncSetAttribute(brx_kernel<23>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(brx_kernel<22>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
    return e;
}

// The products as a tensor of 64-byte pieces (a pair of outputs at a pair of
// points, of two ciphertexts): (16 words, pair of outputs, couple of the tile,
// (tile, pair of points)); a box is a couple's pieces at 16 pairs of points.
// (One ciphertext's 32-byte pieces took 5,000 clocks for the 64 KB.)
static_assert(sizeof(TensorMap) == sizeof(CUtensorMap) && alignof(TensorMap) >= alignof(CUtensorMap), "tensor map");
cudaError_t make_prod_map(Workspace &ws)
{
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found);
    if (e != cudaSuccess) return e;
    if (found != cudaDriverEntryPointSuccess || !fn) return cudaErrorNotSupported;
    const cuuint64_t dims[4] = {16, (cuuint64_t)XN, (cuuint64_t)TILE / 2, TILES * PH};
    const cuuint64_t strides[3] = {32 * TILE, 64, 32 * TILE * XN};  // bytes, of dimensions 1 to 3
    const cuuint32_t box[4] = {16, (cuuint32_t)XN, 1, PH / 2}, step[4] = {1, 1, 1, 1};
    const CUresult r = reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(fn)(
        reinterpret_cast<CUtensorMap *>(&ws.prod_map), CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, ws.prod, dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// (A cooperative launch is checked against the whole device's SMs, so that on
// such a stream its CTAs would wait for ones that cannot start.)
bool limited_stream(cudaStream_t s)
{
    using Query = decltype(&cuStreamGetGreenCtx);
    static const Query query = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        const cudaError_t e = cudaGetDriverEntryPoint("cuStreamGetGreenCtx", &fn, cudaEnableDefault, &found);
        if (e != cudaSuccess) cudaGetLastError();
        return e == cudaSuccess && found == cudaDriverEntryPointSuccess ? reinterpret_cast<Query>(fn) : nullptr;
    }();  // a driver without green contexts: none
    CUgreenCtx ctx = nullptr;
    return query && query(s, &ctx) == CUDA_SUCCESS && ctx;
}

cudaError_t launch(const Workspace &ws, int nsm, const uint32_t *d_lwe2N, const uint64_t *d_luts,
                   const uint32_t *d_lut_id, uint32_t nlut, uint64_t *d_out, size_t B, uint32_t n, uint32_t *d_err,
                   cudaStream_t s, uint32_t mlk, uint32_t pbs_bw, uint32_t tie_rule)
{
    if (B == 0 || B > WAVE) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemsetAsync(ws.sync, 0, SYNC_BYTES, s);
    if (e != cudaSuccess) return e;
    u32 Bu = (u32)B;
    void *args[] = {(void *)&d_lwe2N, (void *)&d_luts, (void *)&d_lut_id, (void *)&nlut, (void *)&ws.weights,
                    (void *)&ws.bsk, (void *)&ws.eval, (void *)&ws.prod, (void *)&ws.acc, (void *)&d_out, (void *)&Bu,
                    (void *)&n, (void *)&d_err, (void *)&mlk, (void *)&tie_rule, (void *)&ws.sync, (void *)&ws.polls, (void *)&ws.prod_map};
    const void *k = pbs_bw == 22 ? (const void *)brx_kernel<22> : (const void *)brx_kernel<23>;
    return cudaLaunchCooperativeKernel(k, dim3((unsigned)nsm), dim3(THREADS), args, SMEM_BYTES, s);
}

}  // namespace brx
}  // namespace luthe
