// Blind rotation of the smallest batches: one ciphertext on a cluster of 2K
// CTAs (K = 4 or 2), one per SM.
//
// A lone ciphertext is a chain of n steps, so its time is the length of a step
// on the SMs that share it.  On two SMs (br_kernel_pair) a step takes 16,400
// clocks, most of it integer issue of 2048-point transforms; here each
// transform is cut into K parts:
//
//   X^2048 + 1 = prod_{h<K} (X^M - w_h),  M = 2048 / K,  w_h = psi^(M (2h+1))
//
// CTA (r, h) owns polynomial (column) r modulo X^M - w_h.  The cut itself is
// sums of shifted digits (w_h is a power of two), and every CTA of a column
// keeps the whole accumulator polynomial and does the rotation, the
// decomposition and the final radix-K sum for itself: they are short, and the
// step is left with two exchanges over distributed shared memory, of M words
// with the CTA of the other column before the product and among the K CTAs of
// the column after the inverse transform.
//
// A part's transform is the plain radix-2 tree (X^L - psi^E into X^(L/2) -+
// psi^(E/2)), two points a thread: log2(M) - 6 levels in small groups of lanes,
// one pass through shared memory, six levels in a warp, the other exchanges
// being shuffles.  All twiddles are per-thread constants in registers.
//
// Bound: a step of K = 4 takes 7,150 clocks (3.72 us), of which about 3,500 in
// the two transforms, 2,300 in the rotation, decomposition and radix-4 sum that
// every CTA of a column repeats, 1,600 in the exchanges.  The integer ALU is
// busy half of the time, two warps to a scheduler cannot fill more.  K = 8
// would halve the transforms only, and few GPCs have room for 16 SMs.
// Measured (n = 804, 148 SMs): 1 to 15 ciphertexts 2.99 to 3.05 ms (K = 4), 16
// to 33 4.34 ms (K = 2), both 6.83 ms on two SMs.
//
// Part of kernels.cu (it shares the bounds of the waits).
#pragma once

namespace luthe {
namespace parts {

constexpr int POINTS = 64;  // of a warp's sub-block
template <int K>
struct Shape {
    static constexpr int M = N / K, T = M / 2, LOG = K == 4 ? 9 : 10;
    static constexpr int SA = LOG - 6, GL = 1 << (SA - 1);  // levels and lanes of the first pass
    static constexpr int PAD = 16 / GL;   // words after every 64 accumulator words: a half-warp's GL runs in different banks
    static constexpr int ROW = POINTS + 8 / GL;  // staging row, same reason
    static constexpr int ACC = N + N / 64 * PAD, STAGE = (M / POINTS) * ROW;
};
static_assert(Shape<4>::T == 256 && Shape<2>::T == 512 && Shape<4>::M / POINTS * 32 == Shape<4>::T, "shape");

template <int K>
struct Shared {
    using S = Shape<K>;
    u64 rx[2][2 * S::T];           // [step parity]: the other column's evaluations, by thread
    u64 ry[2][K][2 * S::T];        // [step parity][part]: inverse transforms of this column, by thread
    u64 acc[S::ACC], fwd[S::STAGE], inv[S::STAGE];
    u64 ex[2], ey[2];              // mbarriers of rx, ry
    u32 sent_x, sent_y;
};

__device__ __forceinline__ u32 remote(u32 addr, u32 rank)
{
    u32 a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}
__device__ __forceinline__ void send2(u32 dst, u64 a, u64 b, u32 mbar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst), "l"(a),
                 "l"(b), "r"(mbar)
                 : "memory");
}
// bounded wait for a phase; what the cluster sent with it is visible after it
__device__ __forceinline__ bool wait_phase(u64 *m, u32 parity, unsigned long long polls)
{
    const u32 a = smem_addr(m);
    for (unsigned long long it = 0; it < polls; it++) {
        u32 done;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(a), "r"(parity)
                     : "memory");
        if (done) return true;
    }
    return false;
}

// Swap between the lanes that differ in `mask`: the lane without that bit holds
// the lower elements of branches 0 (a) and 1 (b) and goes on with branch 0, the
// other one holds the upper elements and goes on with branch 1.  Its own inverse.
__device__ __forceinline__ void swap_lanes(u64 &a, u64 &b, int mask, bool bit)
{
    const u64 r = __shfl_xor_sync(0xFFFFFFFFu, bit ? a : b, mask);
    if (bit) a = r;
    else b = r;
}
// One level down the tree: a + b w and a - b w, w < p.  The sums are taken on
// the 128-bit product (p 2^64 + a - b w is positive), so that a modular add does
// not follow the reduction in the chain.
__device__ __forceinline__ void tree_fwd(u64 &a, u64 &b, u64 w)
{
    u64 lo, hi, l1, h1, l2, h2;
    gl::mul_wide(b, w, lo, hi);
    asm("add.cc.u64 %0, %2, %4;\n\t"
        "addc.u64 %1, %3, 0;"
        : "=l"(l1), "=l"(h1)
        : "l"(lo), "l"(hi), "l"(a));
    asm("sub.cc.u64 %0, %4, %2;\n\t"
        "subc.u64 %1, %5, %3;"
        : "=l"(l2), "=l"(h2)
        : "l"(lo), "l"(hi), "l"(a), "l"(gl::P));
    a = gl::reduce128(l1, h1);
    b = gl::reduce128(l2, h2);
}
// and back: a + b and (a - b) w
__device__ __forceinline__ void tree_inv(u64 &a, u64 &b, u64 w)
{
    const u64 t = gl::sub(a, b);
    a = gl::add(a, b);
    b = gl::mul(t, w);
}
// (l : h) + x y mod p
__device__ __forceinline__ u64 mul_onto(u64 l, u64 h, u64 x, u64 y)
{
    u64 l1, h1;
    u32 c;
    gl::mul_wide(x, y, l1, h1);
    asm("add.cc.u64 %0, %0, %3;\n\t"
        "addc.cc.u64 %1, %1, %4;\n\t"
        "addc.u32 %2, 0, 0;"
        : "+l"(l1), "+l"(h1), "=r"(c)
        : "l"(l), "l"(h));
    return gl::sub(gl::reduce128(l1, h1), (u64)c << 32);  // 2^128 = -2^32
}

// psi^e: 2^(3 (e / 64)) psi^(e mod 64) (tw holds psi^j2 in its first 64 words)
__device__ __forceinline__ u64 psi_pow(const u64 *tw, u32 e)
{
    e &= TWO_N - 1;
    return gl::canon(gl::mul(ntt::c_pow2.v[(3 * (e >> 6)) % 192], tw[e & 63]));
}

// Balanced digit (signed, gl::decomp_to_p) of a torus word by its upper half:
// rounding, sign and wrap are one addition, z / 2^(32-BW) = d + 2^(BW-1); a zero
// quotient is the tie, which is positive from tie_floor on.
template <int BW>
__device__ __forceinline__ int digit(u32 hi, u32 tie_floor)
{
    constexpr u32 RB = 1u << (31 - BW);
    const u32 z = hi + (0x80000000u + RB);
    u32 d = z >> (32 - BW);
    if (z - tie_floor < 2 * RB - tie_floor) d = 1u << BW;
    return (int)(d - (1u << (BW - 1)));
}

// p0 + p1 2^24 + p2 2^48 + p3 2^72 mod p of signed 24-bit p
__device__ __forceinline__ u64 shifted_sum(int p0, int p1, int p2, int p3)
{
    const long long low = (long long)p0 + (long long)p1 * (1 << 24), high = (long long)p2 + (long long)p3 * (1 << 24);
    // high 2^48 = (high mod 2^16) 2^48 + (high >> 16) (2^32 - 1)
    const long long hh = high >> 16, rest = low - hh + (hh << 32);
    return gl::add((u64)high << 48, rest < 0 ? (u64)rest + gl::P : (u64)rest);
}

template <int K, int BW>
__global__ void __cluster_dims__(2 * K, 1, 1) __launch_bounds__(Shape<K>::T, 1)
    br_parts_kernel(const u32 *__restrict__ lwe2N, const u64 *__restrict__ luts, const u32 *__restrict__ lut_id, u32 nlut,
                    const u64 *__restrict__ bsk, const u64 *__restrict__ tw, u64 *__restrict__ out, u32 n,
                    u32 *__restrict__ err, const u32 *__restrict__ dst_idx, u32 mlk, u32 tie_rule)
{
    namespace cg = cooperative_groups;
    using S = Shape<K>;
    cg::cluster_group cluster = cg::this_cluster();
    const u32 rank = cluster.block_rank(), r = rank / K, h = rank % K;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    Shared<K> &sh = *reinterpret_cast<Shared<K> *>(smem_raw);
    const unsigned long long polls = g_slab_wait_polls;
    const u32 tie_floor = tie_rule == TIE_RTL ? 1u << (31 - BW) : 0u;
    const u32 t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const u32 l = t % S::GL, j2 = t / S::GL, x0 = j2 + POINTS * l;  // first pass: points x0 and x0 + M / 2
    const u32 ct = blockIdx.x / (2 * K);
    constexpr u32 SHARE = S::T * 16;  // bytes of one CTA's contribution to an exchange

    if (t == 0) {
        for (int i = 0; i < 2; i++) {
            mbar_init(&sh.ex[i], 1);
            mbar_init(&sh.ey[i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < 2; i++) {
            mbar_expect_tx(&sh.ex[i], SHARE);
            mbar_expect_tx(&sh.ey[i], K * SHARE);
        }
    }

    // twiddles: level L splits X^(M/2^(L-1)) - psi^E by psi^(E/2); the branches taken so far (b_1 first) are the
    // thread's lane bits in the first pass, its thread index bits in the second
    u64 wf[S::LOG], wi[S::LOG];
#pragma unroll
    for (int L = 1; L <= S::LOG; L++) {
        u32 e = (u32)(S::M >> L) * (2 * h + 1);
        const u32 path = L <= S::SA ? l << (S::LOG - 1 - (S::SA - 1)) : t;  // b_1 is bit LOG - 2
#pragma unroll
        for (int i = 1; i < L; i++) e += (path >> (S::LOG - 1 - i) & 1) << (11 - (L - i));
        wf[L - 1] = psi_pow(tw, e);
        wi[L - 1] = psi_pow(tw, TWO_N - (e & (TWO_N - 1)));
    }
    // this thread's two evaluation points k = h + K m, m = the path with b_1 lowest; their BSK words of column r
    u32 m = 0;
#pragma unroll
    for (int i = 1; i < S::LOG; i++) m |= (t >> (S::LOG - 1 - i) & 1) << (i - 1);
    const u64 *bp[2];
#pragma unroll
    for (int e = 0; e < 2; e++) {
        const u32 k = h + K * (m + (e << (S::LOG - 1)));
        bp[e] = bsk + ((u32)ntt::brv3(k >> 8) * 4 + r) * 256 + (k & 255);  // row 0; row 1 is 512 words on
    }

    const u32 *my_lwe = lwe2N + (size_t)ct * (n + 1);
    u32 lid = lut_id[ct];
    if (lid >= nlut) {  // device-resident ids cannot be checked by the host: flag it, stay in bounds
        if (t == 0 && rank == 0) atomicOr(err, DEVERR_LUT_ID);
        lid = 0;
    }
    // accumulator words of this thread: x0 + (M/2) e + M q, at index e K + q
    u64 acc[2 * K];
    u64 *own = sh.acc + x0 + S::PAD * (x0 >> 6);
    constexpr u32 HALF = S::M / 2 + S::PAD * (S::M / 128);  // offset of M/2 words in sh.acc
#pragma unroll
    for (int e = 0; e < 2; e++)
#pragma unroll
        for (int q = 0; q < K; q++) {
            acc[e * K + q] = luts[((size_t)lid * 2 + r) * N + x0 + (S::M / 2) * (e + 2 * q)];
            own[HALF * (e + 2 * q)] = acc[e * K + q];
        }
    u64 b[4], nb[4];  // [point][row: this column's polynomial, the other one]
#pragma unroll
    for (int e = 0; e < 4; e++) b[e] = __ldg(bp[e >> 1] + ((e & 1) ^ r) * 512);
    const u32 peer = rank ^ K;  // the same part of the other column
    const u32 peer_rx = remote(smem_addr(sh.rx) + t * 16, peer), peer_ex = remote(smem_addr(sh.ex), peer);
    cluster.sync();  // every CTA's barriers are set up before any remote access

    u32 sent_x = 0, sent_y = 0, got_x = 0, got_y = 0;  // exchanges sent and received (uniform over the CTA)
    u32 a_next = my_lwe[0];
    bool ok = true;
    u64 y[2];
    for (u32 i = 0; i < n; i++) {
        const u32 a = a_next, par = i & 1, ph = (i >> 1) & 1;
        a_next = my_lwe[i + 1];
#pragma unroll
        for (int e = 0; e < 4; e++) nb[e] = __ldg(bp[e >> 1] + (size_t)min(i + 1, n - 1) * SLAB_WORDS + ((e & 1) ^ r) * 512);
#pragma unroll
        for (int e = 0; e < 2; e++) {
            int d[4] = {0, 0, 0, 0};
#pragma unroll
            for (int q = 0; q < K; q++) {
                const u32 src = x0 + (S::M / 2) * (e + 2 * q) + TWO_N - a, s = src & (N - 1);
                const u64 neg = (src & N) ? ~0ull : 0ull;
                const u64 rot = sh.acc[s + S::PAD * (s >> 6)];
                d[q] = digit<BW>((u32)(((rot ^ neg) - neg - acc[e * K + q]) >> 32), tie_floor);
            }
            if constexpr (K == 4) {
                // sum d_j 2^(24 (2h+1) j): the exponents are 0, 24, 48, 72 in another order, with signs (2^96 = -1)
                const int p1 = h & 1 ? d[3] : d[1], p3 = h & 1 ? d[1] : d[3];
                const int s1 = h >= 2 ? -1 : 1, s2 = h & 1 ? -1 : 1;
                y[e] = shifted_sum(d[0], p1 * s1, d[2] * s2, p3 * s1);
            } else {
                y[e] = shifted_sum(d[0], 0, h ? -d[1] : d[1], 0);
            }
        }
#pragma unroll
        for (int L = 1; L <= S::SA; L++) {
            tree_fwd(y[0], y[1], wf[L - 1]);
            if (L < S::SA) swap_lanes(y[0], y[1], S::GL >> L, l & (S::GL >> L));
        }
        sh.fwd[(2 * l) * S::ROW + j2] = y[0];
        sh.fwd[(2 * l + 1) * S::ROW + j2] = y[1];
        __syncthreads();
        y[0] = sh.fwd[warp * S::ROW + lane];
        y[1] = sh.fwd[warp * S::ROW + lane + 32];
#pragma unroll
        for (int L = S::SA + 1; L <= S::LOG; L++) {
            tree_fwd(y[0], y[1], wf[L - 1]);
            if (L < S::LOG) swap_lanes(y[0], y[1], 16 >> (L - S::SA - 1), lane & (16 >> (L - S::SA - 1)));
        }
        send2(peer_rx + par * (u32)sizeof(sh.rx[0]), y[0], y[1], peer_ex + par * 8);
        sent_x++;
        // the product's own half while the other evaluations are on their way
        u64 lo[2], hi[2];
        gl::mul_wide(y[0], b[0], lo[0], hi[0]);
        gl::mul_wide(y[1], b[2], lo[1], hi[1]);
        ok = wait_phase(&sh.ex[par], ph, polls);
        if (t == 0 && ok) mbar_expect_tx(&sh.ex[par], SHARE);  // for the step after the next
        {
            const ulonglong2 o = *reinterpret_cast<const ulonglong2 *>(&sh.rx[par][2 * t]);
            y[0] = mul_onto(lo[0], hi[0], o.x, b[1]);
            y[1] = mul_onto(lo[1], hi[1], o.y, b[3]);
        }
#pragma unroll
        for (int e = 0; e < 4; e++) b[e] = nb[e];
#pragma unroll
        for (int L = S::LOG; L > S::SA; L--) {
            tree_inv(y[0], y[1], wi[L - 1]);
            if (L > S::SA + 1) swap_lanes(y[0], y[1], 16 >> (L - S::SA - 2), lane & (16 >> (L - S::SA - 2)));
        }
        sh.inv[warp * S::ROW + lane] = y[0];
        sh.inv[warp * S::ROW + lane + 32] = y[1];
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        got_x++;
        y[0] = sh.inv[(2 * l) * S::ROW + j2];
        y[1] = sh.inv[(2 * l + 1) * S::ROW + j2];
#pragma unroll
        for (int L = S::SA; L >= 1; L--) {
            tree_inv(y[0], y[1], wi[L - 1]);
            if (L > 1) swap_lanes(y[0], y[1], S::GL >> (L - 1), l & (S::GL >> (L - 1)));
        }
#pragma unroll
        for (int p = 0; p < K; p++)
            send2(remote(smem_addr(&sh.ry[par][h][2 * t]), r * K + p), y[0], y[1], remote(smem_addr(&sh.ey[par]), r * K + p));
        sent_y++;
        ok = wait_phase(&sh.ey[par], ph, polls);
        if (t == 0 && ok) mbar_expect_tx(&sh.ey[par], K * SHARE);
        {
            u64 v[K][2];
#pragma unroll
            for (int p = 0; p < K; p++) {
                const ulonglong2 o = *reinterpret_cast<const ulonglong2 *>(&sh.ry[par][p][2 * t]);
                v[p][0] = o.x;
                v[p][1] = o.y;
            }
            // c_{x + M j} = w_0^-j sum_p (w_0^-2j)^p v_p
#pragma unroll
            for (int e = 0; e < 2; e++) {
                u64 c[K];
                if constexpr (K == 4) {
                    const u64 e0 = gl::add(v[0][e], v[2][e]), e1 = gl::sub(v[0][e], v[2][e]);
                    const u64 o0 = gl::add(v[1][e], v[3][e]), o1 = gl::shl_abs<48>(gl::sub(v[3][e], v[1][e]));  // 2^-48 = -2^48
                    c[0] = gl::add(e0, o0);
                    c[1] = gl::div2k(gl::add(e1, o1), 24);
                    c[2] = gl::shl_abs<48>(gl::sub(o0, e0));
                    c[3] = gl::shl_abs<24>(gl::sub(o1, e1));  // 2^-72 = -2^24
                } else {
                    c[0] = gl::add(v[0][e], v[1][e]);
                    c[1] = gl::shl_abs<48>(gl::sub(v[1][e], v[0][e]));
                }
#pragma unroll
                for (int q = 0; q < K; q++) {
                    acc[e * K + q] = gl::add_modsw(acc[e * K + q], c[q]);
                    own[HALF * (e + 2 * q)] = acc[e * K + q];
                }
            }
        }
        if (__syncthreads_or(!ok)) {
            ok = false;
            break;
        }
        got_y++;
    }
    __syncthreads();
    if (ok) {
        // sample extract of coefficient 0 (many-LUT: m N / mlk) of X^-b ACC: column 0 the mask, a K-th per part
        const size_t row0 = dst_idx ? dst_idx[ct] : (size_t)ct * mlk;
        const u32 body = my_lwe[n];
        for (u32 f = 0; f < mlk; f++) {
            const u32 rot = (body + f * (N / mlk)) & (TWO_N - 1);
            u64 *o = out + (row0 + f) * (N + 1);
            if (r == 0) {
#pragma unroll
                for (int e = 0; e < 2; e++) {
                    const u32 oi = S::M * h + t + S::T * e;
                    const u32 src = ((oi == 0 ? 0u : (u32)N - oi) + rot) & (TWO_N - 1), s = src & (N - 1);
                    u64 v = sh.acc[s + S::PAD * (s >> 6)];
                    if (src >= (u32)N) v = 0ull - v;
                    __stcs(reinterpret_cast<unsigned long long *>(o) + oi, oi == 0 ? v : 0ull - v);
                }
            } else if (t == 0 && h == 0) {
                const u32 s = rot & (N - 1);
                const u64 v = sh.acc[s + S::PAD * (s >> 6)];
                __stcs(reinterpret_cast<unsigned long long *>(o) + N, rot >= (u32)N ? 0ull - v : v);
            }
        }
    }
    // Every CTA is past its last send.  What was sent and not waited for may
    // still be landing here: only after a wait that ran out, and then at most
    // the next two exchanges of each kind.
    if (t == 0) {
        sh.sent_x = sent_x;
        sh.sent_y = sent_y;
    }
    cluster.sync();
    bool all = ok;
    for (u32 p = 0; p < 2 * K; p++) all = all && *cluster.map_shared_rank(&sh.sent_y, p) == n;
    if (t == 0 && !(all && got_y == n)) {
        bool drained = true;
        for (u32 f = got_x; f < *cluster.map_shared_rank(&sh.sent_x, peer); f++)
            drained &= wait_phase(&sh.ex[f & 1], (f >> 1) & 1, DRAIN_POLLS);
        for (u32 f = got_y; f < got_y + 2; f++) {
            u32 missing = 0;
            for (u32 p = 0; p < K; p++) missing += *cluster.map_shared_rank(&sh.sent_y, r * K + p) <= f ? SHARE : 0;
            if (missing == K * SHARE) break;
            if (missing)
                asm volatile("mbarrier.complete_tx.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(
                                 smem_addr(&sh.ey[f & 1])),
                             "r"(missing)
                             : "memory");
            drained &= wait_phase(&sh.ey[f & 1], (f >> 1) & 1, DRAIN_POLLS);
        }
        atomicOr(err, DEVERR_TIMEOUT | (drained ? 0u : DEVERR_DRAIN));
    }
    cluster.sync();  // no CTA leaves while another may still read its counts
}

template <int K, int BW>
static const void *kernel()
{
    return (const void *)br_parts_kernel<K, BW>;
}
static const void *kernel(int K, uint32_t bw)
{
    return K == 4 ? (bw == 22 ? kernel<4, 22>() : kernel<4, 23>()) : (bw == 22 ? kernel<2, 22>() : kernel<2, 23>());
}

// more than half of an SM's shared memory: one CTA to an SM
constexpr int SMEM_BYTES = 132 * 1024;
static_assert(sizeof(Shared<4>) <= SMEM_BYTES && sizeof(Shared<2>) <= SMEM_BYTES, "shared memory");

static cudaLaunchConfig_t config(int K, size_t count, cudaStream_t s)
{
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3((unsigned)(2 * K * count));
    c.blockDim = dim3((unsigned)(N / K / 2));
    c.dynamicSmemBytes = SMEM_BYTES;
    c.stream = s;
    return c;
}

// attributes, and the ciphertexts that run at the same time
static cudaError_t prepare(int K, int *max_count)
{
    *max_count = 0;
    for (uint32_t bw = 22; bw <= 23; bw++) {
        cudaError_t e = cudaFuncSetAttribute(kernel(K, bw), cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2 * K;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t c = config(K, 1, 0);
    c.attrs = &attr;
    c.numAttrs = 1;
    return cudaOccupancyMaxActiveClusters(max_count, kernel(K, 23), &c);
}

static cudaError_t launch(int K, const uint32_t *d_lwe2N, const uint64_t *d_luts, const uint32_t *d_lut_id, uint32_t nlut,
                   const uint64_t *d_bsk, const uint64_t *d_tw, uint64_t *d_out, size_t count, uint32_t n,
                   uint32_t *d_err, cudaStream_t s, const uint32_t *d_dst_idx, uint32_t mlk, uint32_t pbs_bw,
                   uint32_t tie_rule)
{
    void *args[] = {(void *)&d_lwe2N, (void *)&d_luts, (void *)&d_lut_id,  (void *)&nlut, (void *)&d_bsk,
                    (void *)&d_tw,    (void *)&d_out,  (void *)&n,         (void *)&d_err, (void *)&d_dst_idx,
                    (void *)&mlk,     (void *)&tie_rule};
    const cudaLaunchConfig_t c = config(K, count, s);
    return cudaLaunchKernel(kernel(K, pbs_bw), c.gridDim, c.blockDim, args, c.dynamicSmemBytes, s);
}

}  // namespace parts
}  // namespace luthe
