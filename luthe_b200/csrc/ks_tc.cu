// Key switch on the tensor cores.
//
//   out21[c][x] = [x == n] b21 - sum_{y,z} d_{c,y,z} KSK[y][z][x]  (mod 2^21)
//
// (pep_ks_blram_format.sv:158-172,240-243, pep_ks_mult_node.sv:95-104,
// pep_ks_out_process.sv:276-280,336-341) is a matrix product of signed digits
// (one byte each) by the three bytes of every KSK word, exact in 32-bit sums:
// tcgen05 kind::i8, M = ciphertexts, N = (x, byte), K = (coefficient, level).
//
// The digits are made once, by a kernel of their own, in the operand's layout:
// the product has ten column tiles, and each would make them again.  A product CTA
// takes 256 ciphertexts x 85 outputs (255 of 256 columns; both accumulators
// fill TMEM): per 32 K bytes it moves 16 KB for 256 clocks of MMA, a square
// tile being the one that needs least from L2, which at 41 bytes per clock and
// SM is what bounds it.  Batches with fewer tiles than SMs split K over CTAs
// and add their partial sums into a buffer (32-bit wrap-around sums are exact
// mod 2^21 in any order).
//
// One B200, n = 804, KS 3x6: 16384 BLWEs in 0.55 ms against 10.35 ms with
// dp4a/dp2a on the multiply pipe (per pass of 3584: digits 26 us, product 91 us,
// 450 clocks per K step where L2 would allow 390 and the MMAs 256), 65 BLWEs of
// the 2x7 set 24.6 us against 1.24 ms.
#include <algorithm>

#include "kernels.cuh"
#include "tc.cuh"

namespace luthe {
namespace kstc {

constexpr int TM = 128;                  // rows of one operand tile
constexpr int YB = 32;                   // mask coefficients of one K block: one MMA step per level
constexpr int NBLK = N / YB;
constexpr u32 A_STEP = TM * YB;          // 4 KB: [2][128 rows][16 bytes]
constexpr u32 B_STEP = 256 * YB;         // 8 KB: [2][256 columns][16 bytes]
constexpr int SPS = 2;                   // K steps of one stage: one thread's three copies per 512 clocks of MMA
constexpr int STAGES = 6;
constexpr u32 STAGE_A = SPS * A_STEP, STAGE = 2 * STAGE_A + SPS * B_STEP;
constexpr u32 SM_CTL = STAGES * STAGE;
constexpr u32 SMEM_BYTES = SM_CTL + 256;
constexpr int EPI = 256;                 // epilogue threads, one per row
constexpr int THREADS = EPI + 64;        // + a copy warp and an MMA warp
static_assert(EPI * XT * 4 <= SM_CTL, "the outputs are regrouped in the ring's place");
constexpr unsigned long long POLLS = 1ull << 26;

struct Ctl {
    u64 full[STAGES], empty[STAGES], done;
    u32 tmem, failed;
};
static_assert(sizeof(Ctl) <= 256, "control block");

// Order of the coefficients along K: a warp's word of digits holds coefficients
// l, l + 32, l + 64, l + 96 of a run of 128 (lane l), so that it reads whole rows
// and packs four digits without an exchange; a K block is eight such words.
__device__ __forceinline__ u32 k_coef(u32 blk, u32 slot)
{
    return (blk >> 2) * 128 + (blk & 3) * 8 + (slot >> 2) + (slot & 3) * 32;
}

template <int BL>
__host__ __device__ constexpr u32 fields(u32 v, int count)  // v in each of the lowest fields of BL bits
{
    u32 p = 0;
    for (int i = 0; i < count; i++) p |= v << (BL * i);
    return p;
}
// All balanced digits of a torus word (its upper half) at once, as ks_decomp
// (ks_digits.cuh): digit z is field z of s, less HALF - 1, less field z of e.
// e is the rule of a tie, raw digit + carry = B/2: negative where the raw digit
// above has its top bit; for the top digit (RTL's rule) where its own top bit is
// set and the word is not exactly the tie without a rounding bit.  Adding
// HALF - 1 + e to every field makes the carries those of the decomposition.
template <int BL, int L, bool GEN>
__device__ __forceinline__ void digit_fields(u32 hi, u32 &s, u32 &e)
{
    constexpr int TOT = BL * L;
    const u32 t = hi >> (31 - TOT), c = (t + 1) >> 1;
    e = (c >> (2 * BL - 1)) & fields<BL>(1, L - 1);
    if (!GEN && t != (1u << TOT)) e |= (c >> (BL - 1)) & (1u << (BL * (L - 1)));
    s = c + fields<BL>((1u << (BL - 1)) - 1, L) + e;
}
// byte k of w[j] = byte j of v[k], j < 3
__device__ __forceinline__ void transpose(const u32 (&v)[4], u32 (&w)[3])
{
    const u32 a = __byte_perm(v[0], v[1], 0x5140), b = __byte_perm(v[2], v[3], 0x5140);
    w[0] = __byte_perm(a, b, 0x5410);
    w[1] = __byte_perm(a, b, 0x7632);
    w[2] = __byte_perm(__byte_perm(v[0], v[1], 0x0062), __byte_perm(v[2], v[3], 0x0062), 0x5410);
}
// BITS bits from bit AT of four words whose bytes were transposed, a byte each
template <int AT, int BITS>
__device__ __forceinline__ u32 field4(const u32 (&w)[3])
{
    constexpr u32 ONES = 0x01010101u;
    constexpr int J = AT / 8, O = AT % 8;
    if constexpr (O + BITS <= 8) {
        return (w[J] >> O) & (((1u << BITS) - 1) * ONES);
    } else {
        constexpr int LO = 8 - O;
        return ((w[J] >> O) & (((1u << LO) - 1) * ONES)) | ((w[J + 1] & (((1u << (BITS - LO)) - 1) * ONES)) << LO);
    }
}
template <int BL, int L, int Z = 0>
__device__ __forceinline__ void digit_words(const u32 (&s)[3], const u32 (&e)[3], u32 *d)
{
    if constexpr (Z < L) {
        constexpr u32 ONES = 0x01010101u, BIAS = 0x80 * ONES;  // keeps the bytes' differences from borrowing
        d[Z] = (field4<BL * Z, BL>(s) + (BIAS - ((1u << (BL - 1)) - 1) * ONES) - field4<BL * Z, 1>(e)) ^ BIAS;
        digit_words<BL, L, Z + 1>(s, e, d);
    }
}

// Digits of 32 ciphertexts x 128 coefficients, the operand's layout being [row
// tile][K block][level][half][128 rows][16 bytes].  In shared memory row r of run
// g (K block, half) lies at r ^ g: the eight runs of a warp's words would
// otherwise meet in the same banks.  Bound: the integer ALU, 24 instructions per
// coefficient (26 us per 3584 rows; digit by digit, 50 and six byte stores, 37).
constexpr int DR = 32;
template <int BL, int L, bool GEN>
__global__ void __launch_bounds__(256) digits_kernel(const u64 *__restrict__ in, uint8_t *__restrict__ dig, u32 B)
{
    __shared__ __align__(16) u32 sm[4 * L * 2 * DR * 4];  // [K block][level][half][row][4 words]
    const u32 run = blockIdx.x, row0 = blockIdx.y * DR, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const u32 g = lane >> 2;
#pragma unroll
    for (u32 k = 0; k < DR / 8; k++) {
        const u32 r = warp + 8 * k, c = row0 + r;
        u32 s[4], e[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const u32 hi = c < B ? reinterpret_cast<const u32 *>(in)[2 * ((size_t)c * (N + 1) + run * 128 + 32 * j + lane) + 1] : 0u;
            digit_fields<BL, L, GEN>(hi, s[j], e[j]);
        }
        u32 ts[3], te[3], d[L];
        transpose(s, ts);
        transpose(e, te);
        digit_words<BL, L>(ts, te, d);
#pragma unroll
        for (int z = 0; z < L; z++) sm[((((g >> 1) * L + z) * 2 + (g & 1)) * DR + (r ^ g)) * 4 + (lane & 3)] = d[z];
    }
    __syncthreads();
    // runs of 32 rows x 16 bytes
    uint8_t *dst = dig + ((size_t)(row0 / TM) * NBLK + run * 4) * (L * A_STEP) + (row0 % TM) * 16;
    for (u32 i = threadIdx.x; i < 4 * L * 2 * DR; i += 256) {
        const u32 r = i % DR, half = i / DR % 2, z = i / (2 * DR) % L, blk = i / (2 * DR * L);
        *reinterpret_cast<uint4 *>(dst + (blk * L + z) * A_STEP + half * (TM * 16) + r * 16) =
            reinterpret_cast<const uint4 *>(sm)[i - r + (r ^ (blk * 2 + half))];
    }
}

// KSK [x][coefficient][level] -> column tiles of 85 outputs, [tile][K block]
// [level][half][column 3 (x mod 85) + byte][16 coefficients, in the order of
// k_coef]; the last column of a tile stays zero
__global__ void __launch_bounds__(256) layout_kernel(const u32 *__restrict__ ksk, uint8_t *__restrict__ dst, u32 n, u32 L)
{
    const u32 i = blockIdx.x * 256 + threadIdx.x, per_x = N / 16 * L;
    if (i >= (n + 1) * per_x) return;
    const u32 x = i / per_x, y16 = i % per_x / L, z = i % L;
    const u32 *src = ksk + (size_t)x * N * L + z;
    u32 w[3][4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        w[0][j] = w[1][j] = w[2][j] = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const u32 v = src[k_coef(y16 / 2, (y16 & 1) * 16 + 4 * j + k) * L] & ((1u << KS_W) - 1);
#pragma unroll
            for (int b = 0; b < 3; b++) w[b][j] |= ((v >> (8 * b)) & 0xFF) << (8 * k);
        }
    }
    uint4 *o = reinterpret_cast<uint4 *>(dst + (((size_t)(x / XT) * NBLK + y16 / 2) * L + z) * B_STEP + (y16 & 1) * 4096 +
                                         (x % XT) * 48);
#pragma unroll
    for (int b = 0; b < 3; b++) o[b] = make_uint4(w[b][0], w[b][1], w[b][2], w[b][3]);
}

// KSK [x][k] -> the dp4a form, [group of four rows k][3][xpad]: word 0 the low
// bytes of the rows, words 1 and 2 their upper 13 bits as 16-bit halves
__global__ void __launch_bounds__(256) dp4a_layout_kernel(const u32 *__restrict__ ksk, u32 *__restrict__ dst, u32 n, u32 groups,
                                                          u32 xpad)
{
    const u32 x = blockIdx.x * 128 + (threadIdx.x & 127), g = blockIdx.y * 2 + (threadIdx.x >> 7);
    if (g >= groups) return;
    u32 w[3] = {0, 0, 0};
    if (x <= n) {
        const uint4 v = reinterpret_cast<const uint4 *>(ksk)[(size_t)x * groups + g];
        const u32 M = (1u << KS_W) - 1, r[4] = {v.x & M, v.y & M, v.z & M, v.w & M};
        w[0] = (r[0] & 0xFF) | (r[1] & 0xFF) << 8 | (r[2] & 0xFF) << 16 | r[3] << 24;
        w[1] = r[0] >> 8 | r[1] >> 8 << 16;
        w[2] = r[2] >> 8 | r[3] >> 8 << 16;
    }
#pragma unroll
    for (int p = 0; p < 3; p++) dst[((size_t)g * 3 + p) * xpad + x] = w[p];
}

// grid: (column tiles, pairs of row tiles, K slices)
__global__ void __launch_bounds__(THREADS, 1)
    product_kernel(const u64 *__restrict__ in, const uint8_t *__restrict__ dig, const uint8_t *__restrict__ ksk, u32 L,
                   u32 *__restrict__ out21, u32 *__restrict__ out2N, u32 B, u32 n, u32 *__restrict__ part, u32 xpad,
                   u32 *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t sm[];
    Ctl *ctl = reinterpret_cast<Ctl *>(sm + SM_CTL);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const u32 smem = tc::smem_u32(sm);
    const u32 ntile = blockIdx.x, row0 = blockIdx.y * (2 * TM);
    const bool two = row0 + TM < B;  // a second row tile
    const u32 blk0 = NBLK * blockIdx.z / gridDim.z, blk1 = NBLK * (blockIdx.z + 1) / gridDim.z;
    const u32 steps = (blk1 - blk0) * L, stages = (steps + SPS - 1) / SPS;

    if (tid == 0) {
        for (int i = 0; i < STAGES; i++) {
            tc::mbar_init(&ctl->full[i], 1);
            tc::mbar_init(&ctl->empty[i], 1);
        }
        tc::mbar_init(&ctl->done, 1);
        ctl->failed = 0;
        tc::fence_mbar_init();
    }
    if (warp == EPI / 32) tc::tmem_alloc_512(&ctl->tmem);
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const u32 tmem = ctl->tmem;

    if (tid == EPI) {
        // K steps are contiguous in both operands: (block, level)
        const uint8_t *a0 = dig + ((size_t)(blockIdx.y * 2) * NBLK + blk0) * (L * A_STEP);
        const uint8_t *a1 = a0 + (size_t)NBLK * (L * A_STEP);
        const uint8_t *b = ksk + ((size_t)ntile * NBLK + blk0) * (L * B_STEP);
        u32 k = 0;  // stages
        bool good = true;
        for (; k < stages; k++) {
            const u32 st = k % STAGES, m = min((u32)SPS, steps - k * SPS);
            if (k >= STAGES && !(good = tc::mbar_wait(&ctl->empty[st], (k / STAGES - 1) & 1, POLLS))) break;
            uint8_t *s = sm + st * STAGE;
            tc::mbar_expect_tx(&ctl->full[st], m * ((two ? 2 : 1) * A_STEP + B_STEP));
            tc::bulk_g2s(s, a0 + (size_t)k * STAGE_A, m * A_STEP, &ctl->full[st]);
            if (two) tc::bulk_g2s(s + STAGE_A, a1 + (size_t)k * STAGE_A, m * A_STEP, &ctl->full[st]);
            tc::bulk_g2s(s + 2 * STAGE_A, b + (size_t)k * (SPS * B_STEP), m * B_STEP, &ctl->full[st]);
        }
        if (!good) {  // wait (bounded) for the copies in flight before the CTA may end
            ctl->failed = 1;
            for (u32 i = k > (u32)STAGES ? k - STAGES : 0; i < k; i++)
                if (!tc::mbar_wait(&ctl->full[i % STAGES], (i / STAGES) & 1, POLLS)) atomicOr(err, DEVERR_DRAIN);
        }
    } else if (tid == EPI + 32) {
        const u64 da = tc::desc_plain(smem, TM * 16, 128), db = tc::desc_plain(smem + 2 * STAGE_A, 256 * 16, 128);
        bool ready = false, good = true;
        for (u32 k = 0; k < stages; k++) {
            const u32 st = k % STAGES, nx = (k + 1) % STAGES;
            if (!ready && !(good = tc::mbar_wait(&ctl->full[st], (k / STAGES) & 1, POLLS))) break;
            ready = k + 1 < stages && tc::mbar_test(&ctl->full[nx], ((k + 1) / STAGES) & 1);
            tc::fence_after();
#pragma unroll
            for (u32 j = 0; j < (u32)SPS; j++) {
                if (k * SPS + j >= steps) break;
                const u64 ad = tc::desc_at(da, st * STAGE + j * A_STEP), bd = tc::desc_at(db, st * STAGE + j * B_STEP);
                tc::mma_i8(tmem, ad, bd, tc::idesc_i8(256, true, false), k + j > 0);
                if (two) tc::mma_i8(tmem + 256, tc::desc_at(ad, STAGE_A), bd, tc::idesc_i8(256, true, false), k + j > 0);
            }
            tc::commit(&ctl->empty[st]);
        }
        if (!good) ctl->failed = 1;
        tc::commit(&ctl->done);
        if (!tc::mbar_wait(&ctl->done, 0, POLLS)) atomicOr(err, DEVERR_DRAIN);
    }
    __syncwarp();
    __syncthreads();
    tc::fence_after();
    // accumulators -> sums mod 2^32, regrouped in shared memory so that a warp
    // writes a row's outputs together
    u32 *sums = reinterpret_cast<u32 *>(sm);
    const bool failed = ctl->failed != 0;
    if (failed && tid == 0) atomicOr(err, DEVERR_TIMEOUT);
    if (warp < EPI / 32) {
        const u32 src = tmem + (u32)(tid >> 7) * 256 + ((u32)(tid & 96) << 16);
        if (tid < TM || two) {
#pragma unroll 1
            for (u32 g = 0; g < 6; g++) {  // 48 columns = 16 outputs; the last 16 columns hold 5
                u32 w[3][16];
#pragma unroll
                for (int j = 0; j < 3; j++)
                    if (g < 5 || j == 0) tc::tmem_ld16(src + g * 48 + j * 16, w[j]);
#pragma unroll
                for (int j = 0; j < 3; j++)
                    if (g < 5 || j == 0) tc::tmem_wait16(w[j]);
#pragma unroll
                for (int o = 0; o < 16; o++)
                    if (g < 5 || o < 5)
                        sums[tid * XT + g * 16 + o] = w[(3 * o) / 16][(3 * o) % 16] + (w[(3 * o + 1) / 16][(3 * o + 1) % 16] << 8) +
                                                      (w[(3 * o + 2) / 16][(3 * o + 2) % 16] << 16);
            }
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == EPI / 32) tc::tmem_free_512(tmem);
    if (failed) return;
    const u32 M = (1u << KS_W) - 1;
    for (u32 r = warp; r < 2 * TM; r += THREADS / 32) {
        const u32 c = row0 + r;
        if (c >= B) break;
        for (u32 xl = lane; xl < (u32)XT; xl += 32) {
            const u32 x = ntile * XT + xl;
            if (x > n) break;
            const u32 s = sums[r * XT + xl];
            if (part) {
                atomicAdd(&part[(size_t)c * xpad + x], s);
            } else {
                u32 v = 0u - s;
                if (x == n) {
                    const u64 b = in[(size_t)c * (N + 1) + N];
                    v += (u32)((b >> (64 - KS_W)) + ((b >> (63 - KS_W)) & 1ull));
                }
                v &= M;
                if (out21) out21[(size_t)c * (n + 1) + x] = v;
                out2N[(size_t)c * (n + 1) + x] = ((v >> 9) + ((v >> 8) & 1u)) & (TWO_N - 1);
            }
        }
    }
}

}  // namespace kstc

size_t kstc_ksk_bytes(uint32_t n, uint32_t L) { return (size_t)(n / kstc::XT + 1) * kstc::NBLK * L * kstc::B_STEP; }
size_t kstc_digit_bytes(size_t rows, uint32_t L)
{
    return (rows + kstc::TM - 1) / kstc::TM * kstc::NBLK * (size_t)L * kstc::A_STEP;
}

cudaError_t launch_kstc_layout(const uint32_t *d_ksk, uint8_t *d_dst, uint32_t n, uint32_t L, cudaStream_t s)
{
    cudaError_t e = cudaMemsetAsync(d_dst, 0, kstc_ksk_bytes(n, L), s);
    if (e != cudaSuccess) return e;
    const u32 total = (n + 1) * (N / 16 * L);
    kstc::layout_kernel<<<(total + 255) / 256, 256, 0, s>>>(d_ksk, d_dst, n, L);
    return cudaGetLastError();
}

cudaError_t launch_ks_layout(const uint32_t *d_ksk, uint32_t *d_dst, uint32_t n, uint32_t L, uint32_t xpad, cudaStream_t s)
{
    const u32 groups = N * L / 4;
    kstc::dp4a_layout_kernel<<<dim3(xpad / 128, (groups + 1) / 2), 256, 0, s>>>(d_ksk, d_dst, n, groups, xpad);
    return cudaGetLastError();
}

cudaError_t kstc_set_attributes()
{
    return cudaFuncSetAttribute(kstc::product_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kstc::SMEM_BYTES);
}

template <bool GEN>
static cudaError_t launch_digits(const uint64_t *in, uint8_t *dig, u32 B, uint32_t bl, uint32_t L, cudaStream_t s)
{
    const dim3 grid(N / 128, (B + kstc::DR - 1) / kstc::DR);
    if (bl == 3 && L == 6) kstc::digits_kernel<3, 6, GEN><<<grid, 256, 0, s>>>(in, dig, B);
    else if (bl == 3 && L == 5) kstc::digits_kernel<3, 5, GEN><<<grid, 256, 0, s>>>(in, dig, B);
    else if (bl == 2 && L == 8) kstc::digits_kernel<2, 8, GEN><<<grid, 256, 0, s>>>(in, dig, B);
    else if (bl == 2 && L == 7) kstc::digits_kernel<2, 7, GEN><<<grid, 256, 0, s>>>(in, dig, B);
    else return cudaErrorInvalidValue;
    return cudaGetLastError();
}

cudaError_t launch_keyswitch_tc(const KsTc &t, int nsm, const uint64_t *d_in, uint32_t *d_out21, uint32_t *d_out2N,
                                size_t B, uint32_t n, uint32_t xpad, uint32_t bl, uint32_t L, uint32_t tie_rule,
                                uint32_t *d_err, cudaStream_t s)
{
    const u32 cols = n / kstc::XT + 1;
    for (size_t done = 0; done < B; done += t.rows) {
        const u32 m = (u32)std::min(B - done, t.rows);
        const uint64_t *in = d_in + done * (N + 1);
        u32 *o21 = d_out21 ? d_out21 + done * (n + 1) : nullptr, *o2n = d_out2N + done * (n + 1);
        cudaError_t e = tie_rule == TIE_GENERATOR ? launch_digits<true>(in, t.dig, m, bl, L, s)
                                                  : launch_digits<false>(in, t.dig, m, bl, L, s);
        if (e != cudaSuccess) return e;
        const u32 tiles = cols * ((m + 2 * kstc::TM - 1) / (2 * kstc::TM));
        // few tiles: split K so that every SM has a CTA (a slice keeps two blocks or more)
        const u32 split = m <= KSTC_PART_ROWS ? std::max(1u, std::min((u32)nsm / tiles, (u32)kstc::NBLK / 2)) : 1u;
        kstc::product_kernel<<<dim3(cols, tiles / cols, split), kstc::THREADS, kstc::SMEM_BYTES, s>>>(
            in, t.dig, t.ksk, L, o21, o2n, m, n, split > 1 ? t.part : nullptr, xpad, d_err);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if (split > 1 && (e = launch_ks_finish(in, t.part, o21, o2n, m, n, xpad, s)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace luthe
