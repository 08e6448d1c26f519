// Prefill attention tiles on the 5th generation tensor cores (tcgen05, accumulators in tensor memory), f16 or bf16. Query
// rows are packed (row = token * group + head in group, so the heads that share a kv head also share every K / V tile).
// Three kernels:
//   fa_prefill_tma_kernel<64 | 128>  head dims up to 128, any tensors that tensor maps describe (groups of a power of two):
//              256 rows per work item, tiles by tensor copies. Everything usual runs here.
//   fa_prefill_sm100_kernel2         head dim 128, 1024 rows and more that no map describes: 16-byte chunk copies.
//   fa_prefill_sm100_kernel          the same from 512 rows on: 128 rows per block.
//
// fa_prefill_sm100_kernel: one block = 128 packed query rows of one (batch entry, kv head), head dim 128.
//   warps 0-3  softmax: thread = row. Reads its row of S from tensor memory, keeps the running
//              maximum and sum in registers, writes P (16-bit pairs) back to tensor memory and, when the
//              maximum moved by more than 2^8, rescales its row of O in tensor memory.
//   warp 4     loader: K / V tiles of 64 keys, cp.async 16-byte chunks laid out as the 8 x 16 byte
//              core matrices the tensor core reads without swizzling; two stages.
//   warp 5     issues S = Q K^T (M 128, N 64, 8 k-steps; both operands from shared memory) and
//              O += P V (M 128, N 128, 4 k-steps; P from tensor memory, V from shared memory, N-major),
//              and owns the tensor memory allocation (256 columns: S 64, P 32, O 128).
// Two blocks fit one SM (96 KB of shared memory and 256 of the 512 columns each): while one runs its
// softmax the other runs its matrix products.
//
// Every wait on an mbarrier is bounded; a wait that runs out raises a flag that ends all roles, the
// block frees its tensor memory and the host can read the flag (b200_device_wait_status).
//
// Semantics as fa_dense.cu (candle-core/kernels/flash_attn_impl.h:330-443: FA2-order tiles, bottom
// right aligned windows, zeros for rows without a visible key).
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "fa_params.cuh"

namespace b200 {

constexpr int PF_BM = 128, PF_BN = 64, PF_D = 128, PF_THREADS = 192;
constexpr uint32_t PF_TMEM_COLS = 256, PF_S_COL = 0, PF_P_COL = 64, PF_O_COL = 128;
// shared memory, bytes. K-major operands (Q, K): addr(row, chunk) = (row / 8) * 2048 + chunk * 128 + (row % 8) * 16
// (chunk = 8 elements of the head dim); N-major operand (V): addr(key, chunk) = chunk * 1024 + (key / 8) * 128 + (key % 8) * 16
constexpr uint32_t PF_Q_BYTES = 32768, PF_KT_BYTES = 16384, PF_VT_BYTES = 16384;
constexpr uint32_t PF_SM_Q = 0, PF_SM_K = PF_Q_BYTES, PF_SM_V = PF_SM_K + 2 * PF_KT_BYTES, PF_SM_BAR = PF_SM_V + 2 * PF_VT_BYTES;
constexpr uint32_t PF_SMEM = PF_SM_BAR + 128;
constexpr float PF_LOG2E = 1.4426950408889634f, PF_SLACK = 8.0f;

__device__ int g_wait_failed = 0;  // set when a bounded wait ran out in any kernel of this file

// ---- tcgen05 wrappers -------------------------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// shared memory matrix descriptor, no swizzle: start address, K-direction stride (between core
// matrices that follow one another along the contraction), M/N-direction stride, all in 16-byte units
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t k_stride, uint32_t mn_stride) {
    uint64_t d = (uint64_t)((saddr & 0x3ffffu) >> 4);
    d |= (uint64_t)((k_stride >> 4) & 0x3fffu) << 16;
    d |= (uint64_t)((mn_stride >> 4) & 0x3fffu) << 32;
    d |= 1ull << 46;  // descriptor version of this architecture
    return d;
}
// The same for tiles that a tensor copy wrote with the 128-byte swizzle (rows of 128 bytes, 8-row atoms of 1024 bytes,
// tile base aligned to 1024 bytes): `lbo` is the distance between the two 64-element halves of an M/N-major operand
// (unused for a K-major one), `sbo` the distance between 8-row atoms.
__device__ __forceinline__ uint64_t tc_desc_sw128(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = (uint64_t)((saddr & 0x3ffffu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3fffu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3fffu) << 32;
    d |= 1ull << 46;
    d |= 2ull << 61;  // layout type: 128-byte swizzle
    return d;
}
// one box of a tiled tensor map -> shared memory, completion counted in bytes on `bar`; one destination block
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, int c4, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar)
                 : "memory");
}
// instruction descriptor, kind::f16: f32 accumulator, A and B of one 16-bit type, B N-major or K-major
__host__ __device__ constexpr uint32_t tc_idesc(bool bf16, bool b_n_major, uint32_t m, uint32_t n) {
    return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | ((b_n_major ? 1u : 0u) << 16) | ((n >> 3) << 17) | ((m >> 4) << 24);
}
__device__ __forceinline__ void tc_mma_ss(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem), "l"(a),
                 "l"(b), "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
                 "r"(a_tmem), "l"(b), "r"(idesc), "r"(accumulate)
                 : "memory");
}
// 32 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
          "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
          "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
        "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
                 "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
                 : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void pf_cp16(uint32_t dst, const void *src, bool pred) {
    const int n = pred ? 16 : 0;  // zero fill for rows outside the tile
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
template <bool BF16>
__device__ __forceinline__ uint32_t pf_pack2(float lo, float hi) {
    uint32_t d;
    if (BF16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// ---- packed f32 pairs (fma.rn.f32x2 / add.rn.f32x2) and the three-input maximum ----------------------
__device__ __forceinline__ uint64_t pk2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void upk2(uint64_t v, float &lo, float &hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
__device__ __forceinline__ uint64_t ffma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t fadd2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ float fmax3(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// One row's 64 scores of a tile (raw dot products in sa, sb; the softmax scale sl2 > 0 carries log2 e):
// masks, the row maximum, the decision to move the reference maximum (`need`, with the factor `f` that
// takes O and the running sum to the new reference) and P as 16-bit pairs. Three instructions per score
// besides the exponential: a shared three-input maximum, a packed multiply-add and a packed sum.
template <bool BF16>
__device__ __forceinline__ void pf_softmax_row(uint32_t (&sa)[32], uint32_t (&sb)[32], bool full, int lo_rel, int hi_rel, float sl2, bool first,
                                               float &mref, float &l, bool &need, float &f, uint32_t (&pr)[32]) {
    if (!full) {
        // keys lo_rel <= i < hi_rel of the tile are visible to this row (sa: keys 0-31, sb: keys 32-63)
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            if (!(i >= lo_rel && i < hi_rel)) sa[i] = 0xff800000u;
            if (!(i + 32 >= lo_rel && i + 32 < hi_rel)) sb[i] = 0xff800000u;
        }
    }
    float m0 = fmax3(u2f(sa[0]), u2f(sa[1]), u2f(sb[0])), m1 = u2f(sb[1]);
#pragma unroll
    for (int i = 2; i < 32; i += 2) {
        m0 = fmax3(m0, u2f(sa[i]), u2f(sa[i + 1]));
        m1 = fmax3(m1, u2f(sb[i]), u2f(sb[i + 1]));
    }
    const float mx = fmaxf(m0, m1) * sl2;  // sl2 > 0: the maximum commutes with the scale
    need = false;
    if (first) mref = mx;
    else need = mx > mref + PF_SLACK;
    f = need ? fast_exp2(mref - mx) : 1.0f;
    if (need) {
        mref = mx;
        l *= f;
    }
    const float ms = mref == -INFINITY ? 0.0f : mref;
    const uint64_t sc2 = pk2(sl2, sl2), nm2 = pk2(-ms, -ms);
    uint64_t acc_a = pk2(0.0f, 0.0f), acc_b = acc_a;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float a0, a1, b0, b1;
        upk2(ffma2(pk2(u2f(sa[2 * i]), u2f(sa[2 * i + 1])), sc2, nm2), a0, a1);
        upk2(ffma2(pk2(u2f(sb[2 * i]), u2f(sb[2 * i + 1])), sc2, nm2), b0, b1);
        a0 = fast_exp2(a0);
        a1 = fast_exp2(a1);
        b0 = fast_exp2(b0);
        b1 = fast_exp2(b1);
        acc_a = fadd2(acc_a, pk2(a0, a1));
        acc_b = fadd2(acc_b, pk2(b0, b1));
        pr[i] = pf_pack2<BF16>(a0, a1);
        pr[16 + i] = pf_pack2<BF16>(b0, b1);
    }
    float s0, s1, s2, s3;
    upk2(acc_a, s0, s1);
    upk2(acc_b, s2, s3);
    l += (s0 + s1) + (s2 + s3);
}

// The same for the 128 scores of a tile of 128 keys (four chunks of 32 columns), in pieces: the maximum
// over all four chunks first, then the exponentials of two chunks at a time, so that the first half of P
// is on its way to tensor memory while the second is computed.
__device__ __forceinline__ void pf_mask32(uint32_t (&s)[32], int base, int lo_rel, int hi_rel) {
#pragma unroll
    for (int i = 0; i < 32; ++i)
        if (!(base + i >= lo_rel && base + i < hi_rel)) s[i] = 0xff800000u;
}
__device__ __forceinline__ float pf_max64(const uint32_t (&sa)[32], const uint32_t (&sb)[32]) {
    float m0 = fmax3(u2f(sa[0]), u2f(sa[1]), u2f(sb[0])), m1 = u2f(sb[1]);
#pragma unroll
    for (int i = 2; i < 32; i += 2) {
        m0 = fmax3(m0, u2f(sa[i]), u2f(sa[i + 1]));
        m1 = fmax3(m1, u2f(sb[i]), u2f(sb[i + 1]));
    }
    return fmaxf(m0, m1);
}
__device__ __forceinline__ float pf_max32(const uint32_t (&s)[32]) {
    float m0 = fmax3(u2f(s[0]), u2f(s[1]), u2f(s[2])), m1 = fmax3(u2f(s[3]), u2f(s[4]), u2f(s[5]));
#pragma unroll
    for (int i = 6; i < 30; i += 4) {
        m0 = fmax3(m0, u2f(s[i]), u2f(s[i + 1]));
        m1 = fmax3(m1, u2f(s[i + 2]), u2f(s[i + 3]));
    }
    return fmax3(m0, m1, fmaxf(u2f(s[30]), u2f(s[31])));
}
// 32 scores -> 16 columns of P (16-bit pairs), sums into acc
template <bool BF16>
__device__ __forceinline__ void pf_exp32(const uint32_t (&s)[32], uint64_t sc2, uint64_t nm2, uint64_t &acc, uint32_t (&pr)[16]) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        float a0, a1;
        upk2(ffma2(pk2(u2f(s[2 * i]), u2f(s[2 * i + 1])), sc2, nm2), a0, a1);
        a0 = fast_exp2(a0);
        a1 = fast_exp2(a1);
        acc = fadd2(acc, pk2(a0, a1));
        pr[i] = pf_pack2<BF16>(a0, a1);
    }
}
// bounded wait that also ends when another role gave up; false = give up
__device__ __forceinline__ bool pf_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    for (uint32_t i = 0; i < (1u << 20); ++i) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return true;
        if ((i & 255u) == 255u && *abort_flag) return false;
    }
    return false;
}
// bounded wait that ignores the abort flag: for copies in flight that must land before the block leaves
__device__ __forceinline__ void pf_wait_landed(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < (1u << 16); ++i) {
        uint32_t ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(ok)
                     : "r"(bar), "r"(parity)
                     : "memory");
        if (ok) return;
    }
}

template <bool BF16>
__global__ void __launch_bounds__(PF_THREADS, 2) fa_prefill_sm100_kernel(const FaParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + PF_SM_BAR);
    // barriers: 0,1 kv_full; 2,3 kv_empty; 4 s_full; 5 p_full; 6 o_full; 7 drain
    const uint32_t bar0 = sbase + PF_SM_BAR;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + PF_SM_BAR + 64);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + PF_SM_BAR + 72);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const uint32_t hk = blockIdx.y, b = blockIdx.z, G = p.group;
    uint32_t lq = p.lq, lk = p.lk;
    uint64_t q0 = (uint64_t)b * p.lq, k0 = 0;
    if (p.varlen) {
        q0 = p.cu_q[b];
        lq = p.cu_q[b + 1] - p.cu_q[b];
        k0 = p.cu_k[b];
        lk = p.cu_k[b + 1] - p.cu_k[b];
    }
    const uint32_t R = lq * G;
    // the row tiles with the most keys first
    const uint32_t row0 = (gridDim.x - 1 - blockIdx.x) * PF_BM;
    if (row0 >= R) return;
    // a wait that ran out in an earlier block means something is wrong with the device or this build:
    // later blocks leave at once instead of each waiting out its own limit
    if (*reinterpret_cast<volatile int *>(&g_wait_failed)) return;
    const char *qb = reinterpret_cast<const char *>(p.q);
    const char *kb = reinterpret_cast<const char *>(p.k) + (p.varlen ? k0 * p.k_ss + hk * p.k_sh : b * p.k_sb + hk * p.k_sh) * 2;
    const char *vb = reinterpret_cast<const char *>(p.v) + (p.varlen ? k0 * p.v_ss + hk * p.v_sh : b * p.v_sb + hk * p.v_sh) * 2;
    auto range_of = [&](uint32_t r, long long &lo, long long &hi) {
        const long long i = r / G;
        const long long pos = i + (long long)lk - (long long)lq;
        lo = p.wl >= 0 ? max(pos - p.wl, 0ll) : 0ll;
        hi = p.wr >= 0 ? min(pos + p.wr + 1, (long long)lk) : (long long)lk;
        lo = min(lo, (long long)lk);
        hi = max(hi, lo);
    };
    long long t_lo, t_hi, tmp;
    range_of(row0, t_lo, tmp);
    range_of(min(row0 + PF_BM, R) - 1, tmp, t_hi);
    if (t_hi < t_lo) t_hi = t_lo;
    const int ntiles = (int)((t_hi - t_lo + PF_BN - 1) / PF_BN);

    // ---- set up: barriers, tensor memory, the Q tile
    if (tid == 0) {
        mbar_init(&bars[0], 32);
        mbar_init(&bars[1], 32);
        mbar_init(&bars[2], 1);
        mbar_init(&bars[3], 1);
        mbar_init(&bars[4], 1);
        mbar_init(&bars[5], 128);
        mbar_init(&bars[6], 1);
        mbar_init(&bars[7], 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(PF_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // Q: 128 rows x 16 chunks; lanes 0-7 take the 8 rows of one core matrix, lane / 8 four chunks in a row
    for (int idx = tid; idx < PF_BM * 16; idx += PF_THREADS) {
        const int blk = idx >> 5, l = idx & 31;          // 32 chunks = 4 core matrices per step
        const int grp = blk >> 2, kc = (blk & 3) * 4 + (l >> 3), rr = grp * 8 + (l & 7);
        const uint32_t r = row0 + rr;
        const bool ok = r < R;
        const uint32_t i = ok ? r / G : 0, h = hk * G + (ok ? r % G : 0);
        const uint64_t off = (p.varlen ? (q0 + i) * p.q_ss : b * p.q_sb + i * p.q_ss) + h * p.q_sh;
        pf_cp16(sbase + PF_SM_Q + grp * 2048 + kc * 128 + (rr & 7) * 16, qb + off * 2 + kc * 16, ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 4) {
        // ================================================================ loader
        auto load_tile = [&](int t) {
            const long long j0 = t_lo + (long long)t * PF_BN;
            const uint32_t dk = sbase + PF_SM_K + (t & 1) * PF_KT_BYTES, dv = sbase + PF_SM_V + (t & 1) * PF_VT_BYTES;
            // K: 64 keys x 16 chunks, as Q
#pragma unroll 4
            for (int blk = 0; blk < 32; ++blk) {
                const int grp = blk >> 2, kc = (blk & 3) * 4 + (lane >> 3), rr = grp * 8 + (lane & 7);
                const long long j = j0 + rr;
                const bool ok = j < t_hi;
                pf_cp16(dk + grp * 2048 + kc * 128 + (rr & 7) * 16, kb + (uint64_t)(ok ? j : t_lo) * p.k_ss * 2 + kc * 16, ok);
            }
            // V: per chunk of 8 head dims, 64 keys = 8 core matrices of 8 keys; 32 lanes take 32 keys
#pragma unroll 4
            for (int blk = 0; blk < 32; ++blk) {
                // two neighbouring chunks of 16 keys each per step: every key row gives a whole 32-byte sector
                const int dc = (blk >> 2) * 2 + (lane & 1), key = (blk & 3) * 16 + (lane >> 1);
                const long long j = j0 + key;
                const bool ok = j < t_hi;
                pf_cp16(dv + dc * 1024 + (key >> 3) * 128 + (key & 7) * 16, vb + (uint64_t)(ok ? j : t_lo) * p.v_ss * 2 + dc * 16, ok);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        // Two tiles in flight. A tile is announced as soon as it has landed; only then does the loader
        // wait for the products that free the stage it refills (the issuing warp, in turn, waits for a
        // tile only after it has issued the products of the tile before).
        bool ok = true;
        if (ntiles > 0) load_tile(0);
        if (ntiles > 1) load_tile(1);
        for (int t = 0; t < ntiles && ok; ++t) {
            if (t + 1 < ntiles) asm volatile("cp.async.wait_group 1;" ::: "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(&bars[t & 1]);
            if (t + 2 < ntiles) {
                ok = pf_wait(bar0 + 8 * (2 + (t & 1)), (t >> 1) & 1, abort_flag);  // O += P(t) V(t) has read the stage
                ok = __all_sync(0xffffffffu, ok);
                if (ok) load_tile(t + 2);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (!ok) *abort_flag = 1;
    } else if (warp == 5) {
        // ================================================================ matrix products (one lane issues)
        if (lane == 0) {
            constexpr uint32_t IQK = tc_idesc(BF16, false, PF_BM, PF_BN), IPV = tc_idesc(BF16, true, PF_BM, PF_D);
            bool ok = true;
            auto issue_pv = [&](int t) {  // O += P(t) V(t)
                const uint32_t vs = sbase + PF_SM_V + (t & 1) * PF_VT_BYTES;
#pragma unroll
                for (int ks = 0; ks < PF_BN / 16; ++ks)
                    tc_mma_ts(tmem + PF_O_COL, tmem + PF_P_COL + ks * 8, tc_desc(vs + ks * 256, 128, 1024), IPV, (t > 0 || ks > 0) ? 1u : 0u);
                tc_commit(bar0 + 8 * (2 + (t & 1)));  // the stage is free once these have read it
            };
            for (int t = 0; t < ntiles && ok; ++t) {
                if (t > 0) {
                    ok = pf_wait(bar0 + 8 * 5, (t - 1) & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    issue_pv(t - 1);
                }
                ok = pf_wait(bar0 + 8 * (t & 1), (t >> 1) & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                const uint32_t ks_ = sbase + PF_SM_K + (t & 1) * PF_KT_BYTES;
#pragma unroll
                for (int ks = 0; ks < PF_D / 16; ++ks)
                    tc_mma_ss(tmem + PF_S_COL, tc_desc(sbase + PF_SM_Q + ks * 256, 128, 2048), tc_desc(ks_ + ks * 256, 128, 2048), IQK, ks > 0 ? 1u : 0u);
                tc_commit(bar0 + 8 * 4);
            }
            if (ok && ntiles > 0) {
                ok = pf_wait(bar0 + 8 * 5, (ntiles - 1) & 1, abort_flag);
                if (ok) {
                    tc_fence_after();
                    issue_pv(ntiles - 1);
                    tc_commit(bar0 + 8 * 6);
                }
            }
            if (!ok) {
                *abort_flag = 1;
                // let the products already issued finish before the tensor memory goes
                tc_commit(bar0 + 8 * 7);
                for (uint32_t i = 0; i < (1u << 20); ++i) {
                    uint32_t done;
                    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                                 : "=r"(done)
                                 : "r"(bar0 + 8 * 7), "r"(0u)
                                 : "memory");
                    if (done) break;
                }
            }
        }
        __syncwarp();
    } else {
        // ================================================================ softmax, thread = row
        const uint32_t rr = warp * 32 + lane, r = row0 + rr;
        const bool r_ok = r < R;
        long long r_lo = 0, r_hi = 0;
        if (r_ok) range_of(r, r_lo, r_hi);
        // the tightest bounds over the block's rows decide which tiles need masks
        long long lomax, himin;
        {
            long long a, c2;
            range_of(min(row0 + PF_BM, R) - 1, lomax, a);
            range_of(row0, c2, himin);
            if (row0 + PF_BM > R) himin = -1;  // rows past the sequence: always masked
        }
        const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
        const float sl2 = p.scale * p.kd * PF_LOG2E;
        float mref = -INFINITY, l = 0.0f;
        bool ok = true;
        for (int t = 0; t < ntiles; ++t) {
            ok = pf_wait(bar0 + 8 * 4, t & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            uint32_t sa[32], sb[32];
            tc_ld32(lane_base + PF_S_COL, sa);
            tc_ld32(lane_base + PF_S_COL + 32, sb);
            tc_wait_ld();
            const long long j0 = t_lo + (long long)t * PF_BN;
            const bool full = j0 >= lomax && j0 + PF_BN <= himin && j0 + PF_BN <= t_hi;
            const int lo_rel = r_ok ? (int)max(min(r_lo - j0, (long long)PF_BN), 0ll) : PF_BN;
            const int hi_rel = r_ok ? (int)max(min(min(r_hi, t_hi) - j0, (long long)PF_BN), 0ll) : 0;
            bool need;
            float f;
            uint32_t pr[32];
            pf_softmax_row<BF16>(sa, sb, full, lo_rel, hi_rel, sl2, t == 0, mref, l, need, f, pr);
            if (__any_sync(0xffffffffu, need)) {
                // rows whose maximum moved: O goes to the new reference
#pragma unroll 1
                for (int ch = 0; ch < 4; ++ch) {
                    uint32_t o[32];
                    tc_ld32(lane_base + PF_O_COL + 32 * ch, o);
                    tc_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = f2u(u2f(o[i]) * f);
                    tc_st32(lane_base + PF_O_COL + 32 * ch, o);
                }
                tc_wait_st();
            }
            tc_st32(lane_base + PF_P_COL, pr);
            tc_wait_st();
            tc_fence_before();
            mbar_arrive(&bars[5]);
        }
        if (ok && ntiles > 0) {
            ok = pf_wait(bar0 + 8 * 6, 0, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
        }
        if (!ok) *abort_flag = 1;
        // ---- the row of the output: O / l, or zeros
        const float inv = (ok && ntiles > 0 && l > 0.0f) ? p.vd / l : 0.0f;
        const uint32_t i_tok = r_ok ? r / G : 0, h = hk * G + (r_ok ? r % G : 0);
        uint16_t *orow = reinterpret_cast<uint16_t *>(p.o) + ((q0 + i_tok) * p.hq + h) * PF_D;
        if (ok && ntiles > 0) tc_fence_after();
#pragma unroll 1
        for (int ch = 0; ch < 4; ++ch) {
            uint32_t o[32];
            if (ok && ntiles > 0) {
                tc_ld32(lane_base + PF_O_COL + 32 * ch, o);
                tc_wait_ld();
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = 0u;
            }
            if (r_ok) {
#pragma unroll
                for (int v4 = 0; v4 < 4; ++v4) {
                    uint4 w;
                    w.x = pf_pack2<BF16>(u2f(o[8 * v4]) * inv, u2f(o[8 * v4 + 1]) * inv);
                    w.y = pf_pack2<BF16>(u2f(o[8 * v4 + 2]) * inv, u2f(o[8 * v4 + 3]) * inv);
                    w.z = pf_pack2<BF16>(u2f(o[8 * v4 + 4]) * inv, u2f(o[8 * v4 + 5]) * inv);
                    w.w = pf_pack2<BF16>(u2f(o[8 * v4 + 6]) * inv, u2f(o[8 * v4 + 7]) * inv);
                    *reinterpret_cast<uint4 *>(orow + 32 * ch + 8 * v4) = w;
                }
            }
        }
    }
    // ---- tear down
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(PF_TMEM_COLS) : "memory");
    if (tid == 0 && *abort_flag) atomicExch(&g_wait_failed, 1);
}

// ---------------------------------------------------------------------------------------------
// Two row tiles per block: 256 packed rows share every K / V tile, and the two softmax groups take
// turns with the tensor core (while group A runs its softmax the products of group B execute).
//   16 softmax warps: two threads per row, each with 64 of the 128 scores of a key tile (warps 0-3 / 8-11: rows
//   0-127 (A), first / second half of the tile; warps 4-7 / 12-15: rows 128-255 (B)); the halves exchange their
//   maxima through shared memory once per tile. Twice the warps to hide the latency of the exponentials and of
//   the tensor memory round trips: with one thread per row the softmax of a tile took 3300-4800 cycles and the
//   tensor core sat idle three quarters of the time. Warp 16 loader (two stages of 128 keys), warp 17 issues the
//   products and owns the tensor memory: 512 columns = S_A 128, S_B 128 (P_g overwrites the first 64 columns of
//   S_g once the scores are in registers), O_A 128, O_B 128.
//   Tiles of 128 keys: a tcgen05.mma costs the issuing thread about 90 cycles whatever its shape
//   (measured), so S = Q K^T runs as 8 products of N = 128 instead of 16 of N = 64. One block per SM.
// ---------------------------------------------------------------------------------------------
constexpr int P2_THREADS = 576, P2_ROWS = 256, P2_STAGES = 2, P2_BN = 128, P2_LOADER = 16, P2_ISSUER = 17;
constexpr uint32_t P2_KT_BYTES = 32768, P2_VT_BYTES = 32768;  // 128 keys x 128 dims x 2 bytes
constexpr uint32_t P2_TMEM_COLS = 512;
constexpr uint32_t P2_SM_Q = 0, P2_SM_K = 2 * PF_Q_BYTES, P2_SM_V = P2_SM_K + P2_STAGES * P2_KT_BYTES;
constexpr uint32_t P2_SM_BAR = P2_SM_V + P2_STAGES * P2_VT_BYTES, P2_SM_X = P2_SM_BAR + 256;  // exchange: [2][2][2][128] maxima, [2][2][128] sums
constexpr uint32_t P2_SMEM = P2_SM_X + 6144;
__host__ __device__ constexpr uint32_t p2_s_col(int g) { return 128u * g; }
__host__ __device__ constexpr uint32_t p2_p_col(int g) { return 128u * g; }  // over S_g
__host__ __device__ constexpr uint32_t p2_o_col(int g) { return 256u + 128u * g; }
// barriers
constexpr int B_KF = 0, B_VF = P2_STAGES, B_KE = 2 * P2_STAGES, B_VE = 3 * P2_STAGES, B_S = 4 * P2_STAGES, B_P = B_S + 2, B_O = B_P + 2, B_DRAIN = B_O + 1,
              B_X = B_DRAIN + 1,  // per group: both halves of the rows have published their maxima (or sums)
              B_Q = B_X + 2;      // the Q tile has landed

template <bool BF16>
__global__ void __launch_bounds__(P2_THREADS, 1) fa_prefill_sm100_kernel2(const FaParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + P2_SM_BAR);
    // barriers: k_full, v_full, k_empty, v_empty per stage, s_full and p_full per group, o_full, drain (B_* above)
    const uint32_t bar0 = sbase + P2_SM_BAR;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + P2_SM_BAR + 192);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + P2_SM_BAR + 200);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    const uint32_t hk = blockIdx.y, b = blockIdx.z, G = p.group;
    uint32_t lq = p.lq, lk = p.lk;
    uint64_t q0 = (uint64_t)b * p.lq, k0 = 0;
    if (p.varlen) {
        q0 = p.cu_q[b];
        lq = p.cu_q[b + 1] - p.cu_q[b];
        k0 = p.cu_k[b];
        lk = p.cu_k[b + 1] - p.cu_k[b];
    }
    const uint32_t R = lq * G;
    const uint32_t row0 = (gridDim.x - 1 - blockIdx.x) * P2_ROWS;  // the row tiles with the most keys first
    if (row0 >= R) return;
    if (*reinterpret_cast<volatile int *>(&g_wait_failed)) return;
    const char *qb = reinterpret_cast<const char *>(p.q);
    const char *kb = reinterpret_cast<const char *>(p.k) + (p.varlen ? k0 * p.k_ss + hk * p.k_sh : b * p.k_sb + hk * p.k_sh) * 2;
    const char *vb = reinterpret_cast<const char *>(p.v) + (p.varlen ? k0 * p.v_ss + hk * p.v_sh : b * p.v_sb + hk * p.v_sh) * 2;
    auto range_of = [&](uint32_t r, long long &lo, long long &hi) {
        const long long i = r / G;
        const long long pos = i + (long long)lk - (long long)lq;
        lo = p.wl >= 0 ? max(pos - p.wl, 0ll) : 0ll;
        hi = p.wr >= 0 ? min(pos + p.wr + 1, (long long)lk) : (long long)lk;
        lo = min(lo, (long long)lk);
        hi = max(hi, lo);
    };
    long long t_lo, t_hi, tmp;
    range_of(row0, t_lo, tmp);
    range_of(min(row0 + P2_ROWS, R) - 1, tmp, t_hi);
    if (t_hi < t_lo) t_hi = t_lo;
    const int ntiles = (int)((t_hi - t_lo + P2_BN - 1) / P2_BN);

    if (tid == 0) {
        for (int i = 0; i < P2_STAGES; ++i) {
            mbar_init(&bars[B_KF + i], 32);
            mbar_init(&bars[B_VF + i], 32);
            mbar_init(&bars[B_KE + i], 1);
            mbar_init(&bars[B_VE + i], 1);
        }
        mbar_init(&bars[B_S], 1);
        mbar_init(&bars[B_S + 1], 1);
        mbar_init(&bars[B_P], 256);
        mbar_init(&bars[B_P + 1], 256);
        mbar_init(&bars[B_X], 256);
        mbar_init(&bars[B_X + 1], 256);
        mbar_init(&bars[B_O], 1);
        mbar_init(&bars[B_DRAIN], 1);
        mbar_init(&bars[B_Q], P2_THREADS);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == P2_ISSUER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(P2_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // Q: 256 rows x 16 chunks (two K-major operands of 128 rows). Nobody waits for it here: every thread leaves an
    // asynchronous arrival on the Q barrier, which the issuing thread waits for before its first product, so the first
    // K / V tiles load at the same time.
    for (int idx = tid; idx < P2_ROWS * 16; idx += P2_THREADS) {
        const int blk = idx >> 5, l = idx & 31;
        const int grp = blk >> 2, kc = (blk & 3) * 4 + (l >> 3), rr = grp * 8 + (l & 7);
        const uint32_t r = row0 + rr;
        const bool ok = r < R;
        const uint32_t i = ok ? r / G : 0, h = hk * G + (ok ? r % G : 0);
        const uint64_t off = (p.varlen ? (q0 + i) * p.q_ss : b * p.q_sb + i * p.q_ss) + h * p.q_sh;
        pf_cp16(sbase + P2_SM_Q + grp * 2048 + kc * 128 + (rr & 7) * 16, qb + off * 2 + kc * 16, ok);
    }
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar0 + 8 * B_Q) : "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == P2_LOADER) {
        // ================================================================ loader (16-byte chunks)
        // Per lane constants: the lane's row and chunk inside a step of 32 chunks (K: 8 rows x 4 chunks of one
        // core-matrix row group; V: 16 keys x 2 chunks), so that a copy costs an add or two besides itself.
        const uint64_t k_row8 = 8ull * p.k_ss * 2, v_row16 = 16ull * p.v_ss * 2;           // bytes between steps
        const uint64_t k_lane = (uint64_t)(lane & 7) * p.k_ss * 2 + (uint64_t)(lane >> 3) * 16;
        const uint64_t v_lane = (uint64_t)(lane >> 1) * p.v_ss * 2 + (uint64_t)(lane & 1) * 16;
        const uint32_t k_dst_lane = (uint32_t)(lane >> 3) * 128 + (uint32_t)(lane & 7) * 16;
        const uint32_t v_key = (uint32_t)(lane >> 1);
        const uint32_t v_dst_lane = (uint32_t)(lane & 1) * 2048 + (v_key >> 3) * 128 + (v_key & 7) * 16;
        auto load_k = [&](int t) {
            const long long j0 = t_lo + (long long)t * P2_BN;
            const uint32_t dk = sbase + P2_SM_K + (t % P2_STAGES) * P2_KT_BYTES + k_dst_lane;
            const char *ks = kb + (uint64_t)j0 * p.k_ss * 2 + k_lane;
            if (j0 + P2_BN <= t_hi) {
                // whole tile: step = row group g (8 keys) x chunks 4 q .. 4 q + 3
#pragma unroll 4
                for (int g8 = 0; g8 < 16; ++g8) {
                    const char *src = ks + g8 * k_row8;
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) pf_cp16(dk + g8 * 2048 + q4 * 512, src + q4 * 64, true);
                }
            } else {
                // ragged last tile: rows past the end are zero filled
#pragma unroll 4
                for (int blk = 0; blk < 64; ++blk) {
                    const int g8 = blk >> 2, q4 = blk & 3;
                    const bool ok = j0 + g8 * 8 + (lane & 7) < t_hi;
                    pf_cp16(dk + g8 * 2048 + q4 * 512, ok ? ks + g8 * k_row8 + q4 * 64 : kb, ok);
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar0 + 8 * (B_KF + t % P2_STAGES)) : "memory");
        };
        auto load_v = [&](int t) {
            const long long j0 = t_lo + (long long)t * P2_BN;
            const uint32_t dv = sbase + P2_SM_V + (t % P2_STAGES) * P2_VT_BYTES + v_dst_lane;
            const char *vs = vb + (uint64_t)j0 * p.v_ss * 2 + v_lane;
            if (j0 + P2_BN <= t_hi) {
                // whole tile: step = keys 16 q .. 16 q + 15 x chunks 2 c, 2 c + 1
#pragma unroll 2
                for (int q8 = 0; q8 < 8; ++q8) {
                    const char *src = vs + q8 * v_row16;
#pragma unroll
                    for (int c8 = 0; c8 < 8; ++c8) pf_cp16(dv + c8 * 4096 + q8 * 256, src + c8 * 32, true);
                }
            } else {
#pragma unroll 4
                for (int blk = 0; blk < 64; ++blk) {
                    const int q8 = blk >> 3, c8 = blk & 7;
                    const bool ok = j0 + q8 * 16 + (lane >> 1) < t_hi;
                    pf_cp16(dv + c8 * 4096 + q8 * 256, ok ? vs + q8 * v_row16 + c8 * 32 : vb, ok);
                }
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar0 + 8 * (B_VF + t % P2_STAGES)) : "memory");
        };
        // K and V tiles of 128 keys, two stages each, released separately: the K stage of tile t is free as soon as
        // both S = Q K^T of that tile are done (early in the tile's life), the V stage after both O += P V. Nothing
        // here waits for a copy: every lane leaves an asynchronous arrival on the tile's barrier that fires when its
        // copies have landed.
        bool ok = true;
        for (int t = 0; t < ntiles && ok; ++t) {
            if (t >= P2_STAGES) {
                ok = pf_wait(bar0 + 8 * (B_KE + t % P2_STAGES), ((t / P2_STAGES) - 1) & 1, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            load_k(t);
            if (t >= P2_STAGES) {
                ok = pf_wait(bar0 + 8 * (B_VE + t % P2_STAGES), ((t / P2_STAGES) - 1) & 1, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            load_v(t);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        if (!ok) *abort_flag = 1;
    } else if (warp == P2_ISSUER) {
        // ================================================================ matrix products (one lane issues)
        if (lane == 0) {
            constexpr uint32_t IQK = tc_idesc(BF16, false, PF_BM, P2_BN), IPV = tc_idesc(BF16, true, PF_BM, PF_D);
            bool ok = true;
            auto issue_qk = [&](int g, int t) {  // S_g = Q_g K(t)^T
                const uint32_t ks_ = sbase + P2_SM_K + (t % P2_STAGES) * P2_KT_BYTES, qs_ = sbase + P2_SM_Q + g * PF_Q_BYTES;
#pragma unroll
                for (int ks = 0; ks < PF_D / 16; ++ks)
                    tc_mma_ss(tmem + p2_s_col(g), tc_desc(qs_ + ks * 256, 128, 2048), tc_desc(ks_ + ks * 256, 128, 2048), IQK, ks > 0 ? 1u : 0u);
                tc_commit(bar0 + 8 * (B_S + g));
            };
            auto issue_pv = [&](int g, int t) {  // O_g += P_g(t) V(t)
                const uint32_t vs = sbase + P2_SM_V + (t % P2_STAGES) * P2_VT_BYTES;
#pragma unroll
                for (int ks = 0; ks < P2_BN / 16; ++ks)
                    tc_mma_ts(tmem + p2_o_col(g), tmem + p2_s_col(g) + (ks < 4 ? ks * 8 : 64 + (ks - 4) * 8), tc_desc(vs + ks * 256, 128, 2048), IPV,
                              (t > 0 || ks > 0) ? 1u : 0u);  // P of keys 0-63 / 64-127 sits in the first columns of each half of S
            };
            if (ntiles > 0) {
                ok = pf_wait(bar0 + 8 * B_Q, 0, abort_flag) && pf_wait(bar0 + 8 * B_KF, 0, abort_flag);
                if (ok) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the copies wrote through the generic proxy
                    tc_fence_after();
                    issue_qk(0, 0);
                    issue_qk(1, 0);
                    tc_commit(bar0 + 8 * B_KE);
                }
            }
            for (int t = 0; t < ntiles && ok; ++t) {
                ok = pf_wait(bar0 + 8 * B_P, t & 1, abort_flag) &&  // P_A(t) is in tensor memory, S_A is free
                     pf_wait(bar0 + 8 * (B_VF + t % P2_STAGES), (t / P2_STAGES) & 1, abort_flag);
                if (!ok) break;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tc_fence_after();
                issue_pv(0, t);
                if (t + 1 < ntiles) {
                    ok = pf_wait(bar0 + 8 * (B_KF + (t + 1) % P2_STAGES), ((t + 1) / P2_STAGES) & 1, abort_flag);
                    if (!ok) break;
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    tc_fence_after();
                    issue_qk(0, t + 1);
                }
                ok = pf_wait(bar0 + 8 * (B_P + 1), t & 1, abort_flag);
                if (!ok) break;
                tc_fence_after();
                issue_pv(1, t);
                tc_commit(bar0 + 8 * (B_VE + t % P2_STAGES));  // the V stage is free once both have read it
                if (t + 1 < ntiles) {
                    issue_qk(1, t + 1);
                    tc_commit(bar0 + 8 * (B_KE + (t + 1) % P2_STAGES));  // and the K stage of the next tile
                }
            }
            if (ok && ntiles > 0) tc_commit(bar0 + 8 * B_O);
            if (!ok) {
                *abort_flag = 1;
                tc_commit(bar0 + 8 * B_DRAIN);
                for (uint32_t i = 0; i < (1u << 20); ++i) {
                    uint32_t done;
                    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                                 : "=r"(done)
                                 : "r"(bar0 + 8 * B_DRAIN), "r"(0u)
                                 : "memory");
                    if (done) break;
                }
            }
        }
        __syncwarp();
    } else {
        // ================================================================ softmax, two threads per row
        const int half = warp >> 3, g = (warp >> 2) & 1, w4 = warp & 3;
        const uint32_t g_row0 = row0 + g * PF_BM, rr = w4 * 32 + lane;
        const uint32_t r = g_row0 + rr;
        const bool r_ok = r < R;
        long long r_lo = 0, r_hi = 0;
        if (r_ok) range_of(r, r_lo, r_hi);
        long long lomax = 0, himin = -1;  // a group without rows: every tile masked
        if (g_row0 < R) {
            long long a, c2;
            range_of(min(g_row0 + PF_BM, R) - 1, lomax, a);
            range_of(g_row0, c2, himin);
            if (g_row0 + PF_BM > R) himin = -1;
        }
        const uint32_t lane_base = tmem + ((uint32_t)(w4 * 32) << 16);
        // each half keeps its P inside its own 64 columns of S (first 32 of them), so no half overwrites scores the other still reads
        const uint32_t s_col = p2_s_col(g) + 64 * half, p_col = s_col, o_col = p2_o_col(g) + 64 * half;
        float *xmax = reinterpret_cast<float *>(smem + P2_SM_X);           // [tile & 1][group][half][row]
        float *xsum = reinterpret_cast<float *>(smem + P2_SM_X + 4096);    // [group][half][row]
        const float sl2 = p.scale * p.kd * PF_LOG2E;
        float mref = -INFINITY, l = 0.0f;
        bool ok = true;
        for (int t = 0; t < ntiles; ++t) {
            ok = pf_wait(bar0 + 8 * (B_S + g), t & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const long long j0 = t_lo + (long long)t * P2_BN;
            const bool full = j0 >= lomax && j0 + P2_BN <= himin && j0 + P2_BN <= t_hi;
            int lo_rel = 0, hi_rel = P2_BN;
            if (!full) {
                lo_rel = r_ok ? (int)max(min(r_lo - j0, (long long)P2_BN), 0ll) : P2_BN;
                hi_rel = r_ok ? (int)max(min(min(r_hi, t_hi) - j0, (long long)P2_BN), 0ll) : 0;
            }
            // pass 1: this half's maximum, 32 columns at a time (the scores are read again below: a second
            // tensor memory load is cheaper than 64 registers held across the exchange)
            float hmax;
            {
                uint32_t sa[32];
                tc_ld32(lane_base + s_col, sa);
                tc_wait_ld();
                if (!full) pf_mask32(sa, 64 * half, lo_rel, hi_rel);
                hmax = pf_max32(sa);
                tc_ld32(lane_base + s_col + 32, sa);
                tc_wait_ld();
                if (!full) pf_mask32(sa, 64 * half + 32, lo_rel, hi_rel);
                hmax = fmaxf(hmax, pf_max32(sa));
            }
            // the row's maximum over both halves: through shared memory and the group's exchange barrier
            xmax[(((t & 1) * 2 + g) * 2 + half) * PF_BM + rr] = hmax;
            mbar_arrive(&bars[B_X + g]);
            ok = pf_wait(bar0 + 8 * (B_X + g), t & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            const float mx = fmaxf(hmax, xmax[(((t & 1) * 2 + g) * 2 + (half ^ 1)) * PF_BM + rr]) * sl2;  // sl2 > 0
            bool need = false;
            if (t == 0) mref = mx;
            else need = mx > mref + PF_SLACK;
            const float f = need ? fast_exp2(mref - mx) : 1.0f;
            if (need) {
                mref = mx;
                l *= f;
            }
            if (__any_sync(0xffffffffu, need)) {
                // rows whose maximum moved: this half's 64 columns of O go to the new reference
#pragma unroll 1
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t o[32];
                    tc_ld32(lane_base + o_col + 32 * ch, o);
                    tc_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = f2u(u2f(o[i]) * f);
                    tc_st32(lane_base + o_col + 32 * ch, o);
                }
                tc_wait_st();
            }
            // pass 2: exponentials, 32 scores -> 16 columns of P at a time
            const float ms = mref == -INFINITY ? 0.0f : mref;
            const uint64_t sc2 = pk2(sl2, sl2), nm2 = pk2(-ms, -ms);
            uint64_t acc = pk2(0.0f, 0.0f);
            {
                // P goes over columns 0-31 of this half's scores; columns 32-63 are read after the first store, which
                // does not touch them
                uint32_t sa[32], pr[16];
                tc_ld32(lane_base + s_col, sa);
                tc_wait_ld();
                if (!full) pf_mask32(sa, 64 * half, lo_rel, hi_rel);
                pf_exp32<BF16>(sa, sc2, nm2, acc, pr);
                tc_st16(lane_base + p_col, pr);
                tc_ld32(lane_base + s_col + 32, sa);
                tc_wait_ld();
                if (!full) pf_mask32(sa, 64 * half + 32, lo_rel, hi_rel);
                pf_exp32<BF16>(sa, sc2, nm2, acc, pr);
                tc_st16(lane_base + p_col + 16, pr);
            }
            {
                float a0, a1;
                upk2(acc, a0, a1);
                l += a0 + a1;
            }
            tc_wait_st();
            tc_fence_before();
            mbar_arrive(&bars[B_P + g]);
        }
        if (ok && ntiles > 0) {
            ok = pf_wait(bar0 + 8 * B_O, 0, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
        }
        // the row's sum over both halves
        float ltot = l;
        if (ok) {
            xsum[(g * 2 + half) * PF_BM + rr] = l;
            mbar_arrive(&bars[B_X + g]);
            ok = pf_wait(bar0 + 8 * (B_X + g), ntiles & 1, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) ltot = l + xsum[(g * 2 + (half ^ 1)) * PF_BM + rr];
        }
        if (!ok) *abort_flag = 1;
        const float inv = (ok && ntiles > 0 && ltot > 0.0f) ? p.vd / ltot : 0.0f;
        const uint32_t i_tok = r_ok ? r / G : 0, h = hk * G + (r_ok ? r % G : 0);
        uint16_t *orow = reinterpret_cast<uint16_t *>(p.o) + ((q0 + i_tok) * p.hq + h) * PF_D + 64 * half;
        if (ok && ntiles > 0) tc_fence_after();
#pragma unroll 1
        for (int ch = 0; ch < 2; ++ch) {
            uint32_t o[32];
            if (ok && ntiles > 0) {
                tc_ld32(lane_base + o_col + 32 * ch, o);
                tc_wait_ld();
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = 0u;
            }
            if (r_ok) {
#pragma unroll
                for (int v4 = 0; v4 < 4; ++v4) {
                    uint4 w;
                    w.x = pf_pack2<BF16>(u2f(o[8 * v4]) * inv, u2f(o[8 * v4 + 1]) * inv);
                    w.y = pf_pack2<BF16>(u2f(o[8 * v4 + 2]) * inv, u2f(o[8 * v4 + 3]) * inv);
                    w.z = pf_pack2<BF16>(u2f(o[8 * v4 + 4]) * inv, u2f(o[8 * v4 + 5]) * inv);
                    w.w = pf_pack2<BF16>(u2f(o[8 * v4 + 6]) * inv, u2f(o[8 * v4 + 7]) * inv);
                    *reinterpret_cast<uint4 *>(orow + 32 * ch + 8 * v4) = w;
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == P2_ISSUER) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(P2_TMEM_COLS) : "memory");
    if (tid == 0 && *abort_flag) atomicExch(&g_wait_failed, 1);
}


// ---------------------------------------------------------------------------------------------
// fa_prefill_tma_kernel: everything by tensor copies, one softmax thread per row, head dims up to 128.
//   256 packed rows per work item in two groups of 128 (A: warps 0-3, B: warps 4-7, thread = row, the row's 128 scores of
//   a key tile in registers), warp 8 loads, warps 9 and 10 issue the products of one group each, warp 11 owns the tensor
//   memory: S_A 128, S_B 128 (P_g over the first 64 columns of S_g), O_A HD, O_B HD columns.
// What bounds it: the exponentials (16 per cycle and SM) and, at head dim 128, the products take the same 2 048 cycles per
// tile of 256 x 128 scores; at head dim 64 the exponentials alone do. Hence
//   * one thread per row: the scores are read from tensor memory once, and no maximum crosses a barrier (two threads per
//     row read them twice and met at a barrier in every tile);
//   * the groups' exponentials take turns (head dim 128), so that one group's run under the other's products;
//   * P is handed over in two parts, so the products of the first 96 keys run under the exponentials of the others;
//   * one issuing thread per group: the groups' chains (scores, softmax, products) only meet at the shared stages;
//   * a block goes on to other blocks' items (cluster launch control): the next item's Q and first tiles load and its first
//     scores are formed while the last one's rows leave, and no SM waits for a heavy item that came last.
// Measured (us, causal unless said; before: two threads per row, a block per item; head dims other than 128 on mma.sync,
// sequences of different lengths by 16-byte chunks): B 4, 4096 tokens, 32 / 8 heads of 128: 690 -> 502 (1 094 TFLOP/s); B 1,
// 16 384 tokens: 2 031 -> 1 785 (1 232); 8 x 1000 tokens, 16 heads of 64, no mask: 416 -> 81; 4 x 4096, 16 heads of 64: 1 410 ->
// 237; 2 x 2048, 16 / 4 heads of 96: 417 -> 52; 12 sequences of 100-2960: 654 -> 354. At 16 384 tokens a tile of 256 x 128 takes
// 3 100 cycles (the power limit holds the clock near 1.55 GHz), of which a group spends 1 500 in its exponentials and 1 250
// waiting for its next scores: eight 128 x 128 x 16 products with both operands in shared memory take 840 cycles, not 512.
// Taken back: a polynomial for some of the exponentials (on the multiply-add pipe; degree 5, f32 accurate) made every size
// slower, 531 -> 545 at 2 of 16 pairs, -> 635 at 6.
// A group skips the key tiles that none of its rows sees.
// ---------------------------------------------------------------------------------------------
constexpr int P3_THREADS = 384, P3_ROWS = 256, P3_BN = 128, P3_LOADER = 8, P3_ISSUER = 9, P3_OWNER = 11;
template <int HD>
struct P3 {
    static constexpr int HALVES = HD / 64, STAGES = HD == 128 ? 2 : 4;
    static constexpr uint32_t Q_HALF = P3_ROWS * 128, Q_BYTES = HALVES * Q_HALF;          // [half][row][128 bytes, swizzled]
    static constexpr uint32_t T_HALF = P3_BN * 128, T_BYTES = HALVES * T_HALF;             // a K or V tile, likewise
    static constexpr uint32_t SM_K = Q_BYTES, SM_V = SM_K + STAGES * T_BYTES, SM_OUT = SM_V + STAGES * T_BYTES, SM_BAR = SM_OUT + 8 * 4096, SMEM = SM_BAR + 512;
    // barriers
    static constexpr int KF = 0, VF = STAGES, KE = 2 * STAGES, VE = 3 * STAGES, QF = 4 * STAGES, QE = QF + 1, S = QE + 1, P0 = S + 2, P1 = P0 + 2, O = P1 + 2,
                         DRAIN = O + 2, TK = DRAIN + 2, SR = TK + 8, PV = SR + 2, VT = PV + 2, IF = VT + STAGES, IE = IF + 2, CL = IE + 2, GO = CL + 1, COUNT = GO + 1;
    // Head dim 64 leaves tensor memory for P beside S: the next scores are formed as soon as the last ones are in registers.
    // At 128 P lies over the first columns of S, and the next scores follow the products that read it.
    static constexpr bool EARLY = HD == 64;
    static constexpr bool TURNS = !EARLY;  // the groups' exponentials take turns (see the softmax warps)
    __host__ __device__ static constexpr uint32_t p_col(int g) { return EARLY ? 384u + 64u * g : 128u * g; }
    static_assert(COUNT * 8 <= 464, "barriers");  // then the answer (464), item numbers (480), tensor memory (496), give-up flag (504)
};

// The grid's work: items = (batch entries x kv heads) x row tiles x key splits (p.n_splits). The pairs are taken `hpc` at a time (their keys and
// values stay in L2 together), inside such a chunk the row tiles with the most keys first.
struct P3Grid {
    uint32_t tiles, pairs, hpc, items;
    uint32_t group_log2;  // query heads per kv head (a power of two)
    uint32_t tm_order;  // places of head, key and batch entry in the maps (two bits each): K in bits 0-5, V in bits 8-13
    float lag;  // how far (log 2) a row's reference may stay behind its maximum before O is rescaled
};

struct P3Item {
    uint32_t b, hk, row0, R, gl, split;
    uint64_t q0, k0;
    int lq, lk;
    int t_lo, t_hi;  // the keys that some row of the item sees, within the item's key split
    int ntiles;
};
// the keys [lo, hi) that row r sees
__device__ __forceinline__ void p3_range(const FaParams &p, const P3Item &it, uint32_t r, int &lo, int &hi) {
    const int pos = (int)(r >> it.gl) + it.lk - it.lq;
    lo = p.wl >= 0 && pos > p.wl ? min(pos - p.wl, it.lk) : 0;
    hi = p.wr >= 0 && pos < it.lk - p.wr - 1 ? pos + p.wr + 1 : it.lk;
    hi = max(hi, lo);
}
// work item n; false when it has no rows
__device__ __forceinline__ bool p3_item(const FaParams &p, const P3Grid &gr, uint32_t n, P3Item &it) {
    it.split = 0;
    if (p.n_splits > 1) {
        it.split = n % p.n_splits;
        n /= p.n_splits;
    }
    const uint32_t per = gr.hpc * gr.tiles, chunk = n / per, first = chunk * gr.hpc, width = min(gr.hpc, gr.pairs - first), m = n - chunk * per;
    const uint32_t rank = m / width, pair = first + (m - rank * width);
    it.b = pair / p.hkv;
    it.hk = pair - it.b * p.hkv;
    it.row0 = (gr.tiles - 1 - rank) * P3_ROWS;
    it.gl = gr.group_log2;
    it.lq = (int)p.lq;
    it.lk = (int)p.lk;
    it.q0 = (uint64_t)it.b * p.lq;
    it.k0 = 0;
    if (p.varlen) {
        it.q0 = p.cu_q[it.b];
        it.lq = (int)(p.cu_q[it.b + 1] - p.cu_q[it.b]);
        it.k0 = p.cu_k[it.b];
        it.lk = (int)(p.cu_k[it.b + 1] - p.cu_k[it.b]);
    }
    it.R = (uint32_t)it.lq << it.gl;
    if (it.row0 >= it.R) return false;
    int tmp;
    p3_range(p, it, it.row0, it.t_lo, tmp);
    p3_range(p, it, min(it.row0 + P3_ROWS, it.R) - 1, tmp, it.t_hi);
    it.t_hi = max(it.t_hi, it.t_lo);
    it.ntiles = (it.t_hi - it.t_lo + P3_BN - 1) / P3_BN;
    if (p.n_splits > 1) {  // whole tiles
        const int per = (it.ntiles + (int)p.n_splits - 1) / (int)p.n_splits, first = min((int)it.split * per, it.ntiles);
        it.ntiles = min(per, it.ntiles - first);
        it.t_lo += first * P3_BN;
        it.t_hi = max(min(it.t_hi, it.t_lo + it.ntiles * P3_BN), it.t_lo);
    }
    return true;
}
// the key tiles [t0, t1) of the item that some row of group g sees (empty: t0 == t1), and these keys [lo, hi)
__device__ __forceinline__ void p3_group(const FaParams &p, const P3Item &it, int g, int &t0, int &t1, int &lo, int &hi) {
    t0 = t1 = lo = hi = 0;
    const uint32_t first = it.row0 + g * PF_BM;
    if (first >= it.R || it.ntiles == 0) return;
    int tmp;
    p3_range(p, it, first, lo, tmp);
    p3_range(p, it, min(first + PF_BM, it.R) - 1, tmp, hi);
    lo = max(lo, it.t_lo);
    hi = min(hi, it.t_hi);
    if (hi <= lo) return;
    t0 = (lo - it.t_lo) / P3_BN;
    t1 = (hi - it.t_lo + P3_BN - 1) / P3_BN;
}
// Weights of keys that a row does not see are zero, but zero times an infinity is not. So a group's products over V take only the
// steps of 16 keys that hold some it sees, and where the item's keys end inside such a step the owner warp clears the rest of
// it: true for the item's last tile, at key j0, if what follows is another key (masked for all rows of the item) or
// another sequence; past the end of the tensor the copy brings zeros.
__device__ __forceinline__ bool p3_clears(const FaParams &p, const P3Item &it, int j0) {
    return (p.varlen || it.t_hi < it.lk) && j0 + P3_BN > it.t_hi && ((it.t_hi - j0) & 15) != 0;
}
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(e));
    return e != 0;
}
// tcgen05.wait::ld that also carries the loaded registers, so that nothing that uses them moves in front of it
__device__ __forceinline__ void tc_wait_ld_for(uint32_t (&r)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]),
                   "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]),
                   "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]),
                   "+r"(r[31])
                 :
                 : "memory");
}
// a whole warp waits, and goes on or gives up together
__device__ __forceinline__ bool p3_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    return __all_sync(0xffffffffu, pf_wait(bar, parity, abort_flag));
}
// Asks for a block of the grid that has not started yet (cluster launch control): the answer, 16 bytes, lands in shared memory
// and is counted on `bar`.
__device__ __forceinline__ void clc_try_cancel(uint32_t answer, uint32_t bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(answer), "r"(bar) : "memory");
}
// the x index of the block that was given to this one, or -1 when none was left
__device__ __forceinline__ int clc_answer(uint32_t answer) {
    uint32_t given, x = 0;
    asm volatile(
        "{\n .reg .pred p;\n .reg .b128 a;\n ld.shared.b128 a, [%2];\n clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, a;\n"
        " selp.u32 %1, 1, 0, p;\n @p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, a;\n}"
        : "+r"(x), "=r"(given)
        : "r"(answer)
        : "memory");
    return given ? (int)x : -1;
}

template <int HD, bool BF16>
__global__ void __launch_bounds__(P3_THREADS, 1) fa_prefill_tma_kernel(const FaParams p, const __grid_constant__ CUtensorMap tm_k,
                                                                       const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_q,
                                                                       const P3Grid gr) {
    using C = P3<HD>;
    constexpr int NS = C::STAGES;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t sbase = smem_u32(smem), bar0 = sbase + C::SM_BAR;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + C::SM_BAR);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + C::SM_BAR + 496);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + C::SM_BAR + 504);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (*reinterpret_cast<volatile int *>(&g_wait_failed)) return;
    if (tid == 0) {
        for (int i = 0; i < NS; ++i) {
            mbar_init(&bars[C::KF + i], 1);
            mbar_init(&bars[C::VF + i], 1);
            mbar_init(&bars[C::KE + i], 2);
            mbar_init(&bars[C::VE + i], 2);
            mbar_init(&bars[C::VT + i], 1);
        }
        mbar_init(&bars[C::QF], 1);
        mbar_init(&bars[C::QE], 2);
        for (int g = 0; g < 2; ++g) {
            mbar_init(&bars[C::S + g], 1);
            mbar_init(&bars[C::P0 + g], 4);
            mbar_init(&bars[C::P1 + g], 4);
            mbar_init(&bars[C::O + g], 1);
            mbar_init(&bars[C::DRAIN + g], 1);
            mbar_init(&bars[C::SR + g], 4);
            mbar_init(&bars[C::PV + g], 1);
        }
        for (int i = 0; i < 8; ++i) mbar_init(&bars[C::TK + i], 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars[C::IF + i], 1);
            mbar_init(&bars[C::IE + i], 11);  // loader, two issuers, eight softmax warps
        }
        mbar_init(&bars[C::CL], 1);
        mbar_init(&bars[C::GO], 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == P3_OWNER) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool ok = true;
    volatile int *items = reinterpret_cast<volatile int *>(smem + C::SM_BAR + 480);
    // the block's k-th work item, as the owner warp announces it; false: there is none (or a wait has run out)
    auto next_item = [&](int k, int &n) {
        if (!ok || !(ok = p3_wait(bar0 + 8 * (C::IF + (k & 1)), (k >> 1) & 1, abort_flag))) return false;
        n = items[k & 1];
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[C::IE + (k & 1)]);
        return n >= 0;
    };

    if (warp >= 8) {
        // 128 threads x 56 + 256 x 224 = the launch's 384 x 168 registers
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == P3_LOADER) {
            // ============================================================ loader
            uint32_t kv = 0, nq = 0;  // key tiles and Q tiles so far
            uint32_t tail = 0, tail_n = 0;  // a bit per stage: its V tile lands on the tail's barrier; the parity of that barrier's last copy
            const uint64_t k_total = p.varlen ? p.cu_k[p.b] : 0;
            const char *kbase = reinterpret_cast<const char *>(p.k), *vbase = reinterpret_cast<const char *>(p.v);
            for (int k = 0, n; next_item(k, n); ++k) {
                P3Item it;
                p3_item(p, gr, n, it);
                if (it.ntiles == 0) {
                    if (lane == 0) mbar_arrive(&bars[C::GO]);
                    continue;
                }
                auto load = [&](const CUtensorMap *map, uint32_t ord, uint32_t dst, int j, uint32_t bar) {
                    const uint32_t ph = ord & 3u, pk = (ord >> 2) & 3u;
                    const int bb = p.varlen ? 0 : (int)it.b;
                    const int c1 = ph == 0 ? (int)it.hk : (pk == 0 ? j : bb), c2 = ph == 1 ? (int)it.hk : (pk == 1 ? j : bb),
                              c3 = ph == 2 ? (int)it.hk : (pk == 2 ? j : bb);
                    for (int hf = 0; hf < C::HALVES; ++hf) tma_load_4d(dst + hf * C::T_HALF, map, 64 * hf, c1, c2, c3, bar);
                };
                if (nq > 0 && !(ok = p3_wait(bar0 + 8 * C::QE, (nq - 1) & 1, abort_flag))) break;
                if (lane == 0) {
                    // Q: coordinates (element, head in group, kv head, token, batch entry); a box is 64 elements of all heads of
                    // the group for 256 / G tokens = 256 packed rows (row = token * G + head)
                    mbar_expect_tx(&bars[C::QF], C::Q_BYTES);
                    const int tok = (int)((p.varlen ? it.q0 : 0) + (it.row0 >> it.gl));
                    for (int hf = 0; hf < C::HALVES; ++hf)
                        tma_load_5d(sbase + hf * C::Q_HALF, &tm_q, 64 * hf, 0, (int)it.hk, tok, p.varlen ? 0 : (int)it.b, bar0 + 8 * C::QF);
                }
                __syncwarp();
                ++nq;
                for (int t = 0; t < it.ntiles; ++t, ++kv) {
                    const int st = kv % NS, j0 = it.t_lo + t * P3_BN;
                    const uint32_t ph = ((kv / NS) - 1) & 1, dk = sbase + C::SM_K + st * C::T_BYTES, dv = sbase + C::SM_V + st * C::T_BYTES;
                    if (p.varlen && it.k0 + j0 + P3_BN > k_total) {
                        // the end of the last sequence: its rows alone, by 16-byte chunks in the layout of the tensor copies
                        if (kv >= NS && !(ok = p3_wait(bar0 + 8 * (C::KE + st), ph, abort_flag) && p3_wait(bar0 + 8 * (C::VE + st), ph, abort_flag))) break;
                        const char *kr = kbase + ((it.k0 + j0) * p.k_ss + it.hk * p.k_sh) * 2, *vr = vbase + ((it.k0 + j0) * p.v_ss + it.hk * p.v_sh) * 2;
                        const int rows = it.t_hi - j0;
                        for (int idx = lane; idx < P3_BN * HD / 8; idx += 32) {
                            const int row = idx / (HD / 8), ch = idx % (HD / 8);
                            const bool in = row < rows && (uint32_t)ch * 8 < p.d;
                            const uint32_t at = (ch >> 3) * C::T_HALF + row * 128 + (((ch & 7) ^ (row & 7)) << 4);
                            pf_cp16(dk + at, in ? kr + (uint64_t)row * p.k_ss * 2 + ch * 16 : kr, in);
                            pf_cp16(dv + at, in ? vr + (uint64_t)row * p.v_ss * 2 + ch * 16 : vr, in);
                        }
                        asm volatile("cp.async.commit_group;" ::: "memory");
                        asm volatile("cp.async.wait_group 0;" ::: "memory");
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive(&bars[C::KF + st]);
                            mbar_arrive(&bars[C::VF + st]);
                            tail &= ~(1u << st);
                        }
                        continue;
                    }
                    if (kv >= NS && !(ok = p3_wait(bar0 + 8 * (C::KE + st), ph, abort_flag))) break;
                    if (lane == 0) {
                        mbar_expect_tx(&bars[C::KF + st], C::T_BYTES);
                        load(&tm_k, gr.tm_order & 0x3fu, dk, (int)it.k0 + j0, bar0 + 8 * (C::KF + st));
                    }
                    __syncwarp();
                    if (kv >= NS && !(ok = p3_wait(bar0 + 8 * (C::VE + st), ph, abort_flag))) {
                        if (lane == 0) pf_wait_landed(bar0 + 8 * (C::KF + st), (kv / NS) & 1);
                        break;
                    }
                    if (lane == 0) {
                        const int full = p3_clears(p, it, j0) ? C::VT + st : C::VF + st;
                        mbar_expect_tx(&bars[full], C::T_BYTES);
                        load(&tm_v, (gr.tm_order >> 8) & 0x3fu, dv, (int)it.k0 + j0, bar0 + 8 * full);
                        tail = full == C::VT + st ? tail | 1u << st : tail & ~(1u << st);
                        if (full == C::VT + st) tail_n ^= 1u << st;
                    }
                    __syncwarp();
                }
                if (lane == 0) mbar_arrive(&bars[C::GO]);
            }
            if (!ok) {
                // gave up: the copies already issued must land before the block may leave (bounded)
                *abort_flag = 1;
                if (lane == 0) {
                    if (nq > 0) pf_wait_landed(bar0 + 8 * C::QF, (nq - 1) & 1);
                    for (uint32_t t = kv > NS ? kv - NS : 0; t < kv; ++t) {
                        pf_wait_landed(bar0 + 8 * (C::KF + t % NS), (t / NS) & 1);
                        const uint32_t st = t % NS;
                        if (tail >> st & 1u) pf_wait_landed(bar0 + 8 * (C::VT + st), (tail_n >> st & 1u) ^ 1u);
                        else pf_wait_landed(bar0 + 8 * (C::VF + st), (t / NS) & 1);
                    }
                }
            }
        } else if (warp == P3_OWNER) {
            // ============================================================ work items; rows behind the keys of an item
            // The grid has a block per item. A block starts with its own and then takes over blocks that have not started
            // (heaviest first), so that late items go where there is time; items without rows end here. It asks when the last
            // tile of an item has been requested: the answer comes while the tiles in flight are worked on (asked for at an item's
            // start, the early blocks claim too much: 181 against 142 us for 512 items of 1 to 32 tiles).
            const uint64_t k_total = p.varlen ? p.cu_k[p.b] : 0;
            uint32_t kv = 0, asked = 0, parity = 0;  // parity: of each stage's tail barrier, a bit each
            P3Item it, ahead;
            int n = (int)blockIdx.x;
            auto take = [&](P3Item &x) {  // the next block's item, if there is one with rows
                for (;;) {
                    if (lane == 0) {
                        mbar_expect_tx(&bars[C::CL], 16);
                        clc_try_cancel(sbase + C::SM_BAR + 464, bar0 + 8 * C::CL);
                    }
                    __syncwarp();
                    if (!(ok = p3_wait(bar0 + 8 * C::CL, asked++ & 1, abort_flag))) {
                        if (lane == 0) pf_wait_landed(bar0 + 8 * C::CL, (asked - 1) & 1);
                        n = -1;
                        return;
                    }
                    n = clc_answer(sbase + C::SM_BAR + 464);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // read before the next answer is written
                    __syncwarp();
                    if (n < 0 || p3_item(p, gr, (uint32_t)n, x)) return;
                }
            };
            auto announce = [&](int k) {
                if (k >= 2 && !(ok = ok && p3_wait(bar0 + 8 * (C::IE + (k & 1)), ((k >> 1) - 1) & 1, abort_flag))) return;
                if (lane == 0) {
                    items[k & 1] = n;
                    mbar_arrive(&bars[C::IF + (k & 1)]);
                }
                __syncwarp();
            };
            if (!p3_item(p, gr, (uint32_t)n, it)) take(it);
            announce(0);
            for (int k = 1; ok && n >= 0; ++k, it = ahead) {
                if (!(ok = p3_wait(bar0 + 8 * C::GO, (k - 1) & 1, abort_flag))) break;
                take(ahead);
                announce(k);
                if (!ok || it.ntiles == 0) continue;
                kv += it.ntiles;
                const int st = (kv - 1) % NS, j0 = it.t_lo + (it.ntiles - 1) * P3_BN;
                if (!p3_clears(p, it, j0) || (p.varlen && it.k0 + j0 + P3_BN > k_total)) continue;
                // cleared before V is announced
                if (!(ok = p3_wait(bar0 + 8 * (C::VT + st), (parity >> st) & 1, abort_flag))) break;
                parity ^= 1u << st;
                for (int idx = (it.t_hi - j0) * 8 + lane; idx < (it.t_hi - j0 + 15) / 16 * 128; idx += 32)
#pragma unroll
                    for (int hf = 0; hf < C::HALVES; ++hf)
                        *reinterpret_cast<uint4 *>(smem + C::SM_V + st * C::T_BYTES + hf * C::T_HALF + idx * 16) = make_uint4(0, 0, 0, 0);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[C::VF + st]);
            }
            if (!ok) *abort_flag = 1;
        } else {
            // ============================================================ matrix products of group g
            const int g = warp - P3_ISSUER;
            constexpr uint32_t IQK = tc_idesc(BF16, false, PF_BM, P3_BN), IPV = tc_idesc(BF16, true, PF_BM, HD);
            const uint32_t s_t = tmem + 128u * g, p_t = tmem + C::p_col(g), o_t = tmem + 256u + (uint32_t)HD * g;
            const int nks = (int)(p.d + 15) / 16;  // steps of 16 along the head dim that hold anything
            const uint64_t q_desc = tc_desc_sw128(sbase + g * (C::Q_HALF / 2), 16, 1024);
            uint32_t kv = 0, nq = 0, sc = 0;
            // S_g = Q_g K^T of the tile in stage st
            auto scores = [&](int st, bool last) {
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t k_desc = tc_desc_sw128(sbase + C::SM_K + st * C::T_BYTES, 16, 1024);
#pragma unroll
                    for (int ks = 0; ks < HD / 16; ++ks)
                        if (ks < nks)
                            tc_mma_ss(s_t, q_desc + (uint64_t)(((ks >> 2) * C::Q_HALF + (ks & 3) * 32) >> 4),
                                      k_desc + (uint64_t)(((ks >> 2) * C::T_HALF + (ks & 3) * 32) >> 4), IQK, ks > 0 ? 1u : 0u);
                    tc_commit(bar0 + 8 * (C::S + g));
                    tc_commit(bar0 + 8 * (C::KE + st));
                    if (last) tc_commit(bar0 + 8 * C::QE);
                }
                __syncwarp();
            };
            for (int k = 0, n; next_item(k, n); ++k) {
                P3Item it;
                p3_item(p, gr, n, it);
                if (it.ntiles == 0) continue;
                int t0, t1, lo, hi;
                p3_group(p, it, g, t0, t1, lo, hi);
                // the steps of 16 keys that O_g += P_g V takes: all eight, but the first tile starts at the one in the low four bits and the
                // last ends before the one above them
                const int steps = (((lo - it.t_lo) >> 4) - 8 * t0) | (((hi - it.t_lo + 15) >> 4) - 8 * (t1 - 1)) << 4;
                if (!(ok = p3_wait(bar0 + 8 * C::QF, nq & 1, abort_flag))) break;
                ++nq;
                if (t0 == t1 && elect_one()) mbar_arrive(&bars[C::QE]);
                __syncwarp();
                for (int t = 0; t < it.ntiles; ++t, ++kv) {
                    const int st = kv % NS;
                    const uint32_t ph = (kv / NS) & 1;
                    if (t < t0 || t >= t1) {  // a tile that only the other group needs
                        if (!(ok = p3_wait(bar0 + 8 * (C::KF + st), ph, abort_flag))) break;
                        if (elect_one()) mbar_arrive(&bars[C::KE + st]);
                        __syncwarp();
                        if (!(ok = p3_wait(bar0 + 8 * (C::VF + st), ph, abort_flag))) break;
                        if (elect_one()) mbar_arrive(&bars[C::VE + st]);
                        __syncwarp();
                        continue;
                    }
                    // S_g(t): behind O_g += P_g V(t - 1), which reads P out of S_g's columns, or (EARLY) one tile ahead
                    if (!C::EARLY || t == t0) {
                        if (!(ok = p3_wait(bar0 + 8 * (C::KF + st), ph, abort_flag))) break;
                        scores(st, t == t1 - 1);
                    }
                    if (C::EARLY && t + 1 < t1) {
                        const int sn = (kv + 1) % NS;
                        ok = p3_wait(bar0 + 8 * (C::SR + g), sc & 1, abort_flag) && p3_wait(bar0 + 8 * (C::KF + sn), ((kv + 1) / NS) & 1, abort_flag);
                        if (!ok) break;
                        scores(sn, t + 1 == t1 - 1);
                    }
                    const uint64_t v_desc = tc_desc_sw128(sbase + C::SM_V + st * C::T_BYTES, C::T_HALF, 1024);
                    const bool whole = (t != t0 || (steps & 15) == 0) && (t != t1 - 1 || steps >> 4 == 8);
                    auto some = [&](int from, int to) {  // a tile of which steps are left out
                        const int ks0 = t == t0 ? steps & 15 : 0, ks1 = t == t1 - 1 ? steps >> 4 : 8;
#pragma unroll 1
                        for (int ks = max(from, ks0); ks < min(to, ks1); ++ks) tc_mma_ts(o_t, p_t + ks * 8, v_desc + (uint64_t)(ks * 128), IPV, t > t0 || ks > ks0 ? 1u : 0u);
                    };
                    ok = p3_wait(bar0 + 8 * (C::VF + st), ph, abort_flag) && p3_wait(bar0 + 8 * (C::P0 + g), sc & 1, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    if (elect_one()) {  // O_g += P_g(t) V(t): the first 96 keys while the others' exponentials run
                        if (whole) {
#pragma unroll
                            for (int ks = 0; ks < 6; ++ks) tc_mma_ts(o_t, p_t + ks * 8, v_desc + (uint64_t)(ks * 2048 >> 4), IPV, (t > t0 || ks > 0) ? 1u : 0u);
                        } else {
                            some(0, 6);
                        }
                    }
                    __syncwarp();
                    if (!(ok = p3_wait(bar0 + 8 * (C::P1 + g), sc & 1, abort_flag))) break;
                    tc_fence_after();
                    if (elect_one()) {
                        if (whole) {
#pragma unroll
                            for (int ks = 6; ks < 8; ++ks) tc_mma_ts(o_t, p_t + ks * 8, v_desc + (uint64_t)(ks * 2048 >> 4), IPV, 1u);
                        } else {
                            some(6, 8);
                        }
                        tc_commit(bar0 + 8 * (C::VE + st));
                        if (C::EARLY) tc_commit(bar0 + 8 * (C::PV + g));
                        if (t == t1 - 1) tc_commit(bar0 + 8 * (C::O + g));
                    }
                    __syncwarp();
                    ++sc;
                }
            }
            if (!ok) {
                *abort_flag = 1;
                // let the products already issued finish before the tensor memory goes
                if (elect_one()) {
                    tc_commit(bar0 + 8 * (C::DRAIN + g));
                    pf_wait_landed(bar0 + 8 * (C::DRAIN + g), 0);
                }
                __syncwarp();
            }
        }
    } else {
        // ================================================================ softmax, thread = row
        asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        const int g = warp >> 2, w4 = warp & 3;
        const uint32_t lane_base = tmem + ((uint32_t)(w4 * 32) << 16), s_col = lane_base + 128u * g, p_col = lane_base + C::p_col(g), o_col = lane_base + 256u + (uint32_t)HD * g;
        const float sl2 = p.scale * p.kd * PF_LOG2E;
        uint32_t sc = 0, oc = 0, tk = 0;
        P3Item it;
        int n, t0, t1, r_lo, r_hi, lomax, himin;
        // work item k: the group's key tiles, the row's keys and the tightest bounds over the group's rows, from the item's
        // first key on
        auto begin = [&](int k) {
            if (!next_item(k, n)) return false;
            p3_item(p, gr, (uint32_t)n, it);
            int lo, hi, tmp;
            p3_group(p, it, g, t0, t1, lo, hi);
            const uint32_t g_row0 = it.row0 + g * PF_BM, r = g_row0 + w4 * 32 + lane;
            r_lo = r_hi = lomax = 0, himin = -1;
            if (t1 > t0) {
                if (r < it.R) {
                    p3_range(p, it, r, lo, hi);
                    r_lo = lo - it.t_lo;
                    r_hi = min(hi, it.t_hi) - it.t_lo;
                }
                p3_range(p, it, min(g_row0 + PF_BM, it.R) - 1, lo, tmp);
                p3_range(p, it, g_row0, tmp, hi);
                lomax = lo - it.t_lo;
                himin = g_row0 + PF_BM > it.R ? -1 : min(hi, it.t_hi) - it.t_lo;
            }
            return true;
        };
        bool more = begin(0);
        for (int k = 1; more && ok; ++k) {
            float mref = -INFINITY, l = 0.0f;
            for (int t = 0; t < it.ntiles; ++t) {
                const bool mine = t >= t0 && t < t1;
                // The groups' exponentials take turns, A(0) B(0) A(1) B(1) ... (warp w4 of A and warp w4 of B share an SM
                // quadrant): left alone, both groups end up computing exponentials at the same time, at half the rate each, and
                // waiting for their products at the same time. Not where the scores come early: there nobody waits.
                auto my_turn = [&]() { return g == 0 ? (tk == 0 || p3_wait(bar0 + 8 * (C::TK + w4), (tk - 1) & 1, abort_flag)) : p3_wait(bar0 + 8 * (C::TK + 4 + w4), tk & 1, abort_flag); };
                auto pass_turn = [&]() { if (lane == 0) mbar_arrive(&bars[C::TK + (g ^ 1) * 4 + w4]); };
                if (!mine) {
                    if (C::TURNS) {
                        if (!(ok = my_turn())) break;
                        pass_turn();
                        ++tk;
                    }
                    continue;
                }
                if (!(ok = p3_wait(bar0 + 8 * (C::S + g), sc & 1, abort_flag))) break;
                tc_fence_after();
                uint32_t s0[32], s1[32], s2[32], s3[32];
                tc_ld32(s_col, s0);
                tc_ld32(s_col + 32, s1);
                tc_wait_ld_for(s0);
                tc_wait_ld_for(s1);
                tc_ld32(s_col + 64, s2);
                tc_ld32(s_col + 96, s3);
                const int j0 = t * P3_BN;  // from the item's first key
                const bool full = j0 >= lomax && j0 + P3_BN <= himin;
                const int lo_rel = r_lo - j0, hi_rel = r_hi - j0;
                if (!full) {
                    pf_mask32(s0, 0, lo_rel, hi_rel);
                    pf_mask32(s1, 32, lo_rel, hi_rel);
                }
                const float mx01 = pf_max64(s0, s1);
                tc_wait_ld_for(s2);
                tc_wait_ld_for(s3);
                if (C::EARLY) {  // the scores are in registers: the next ones may come
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&bars[C::SR + g]);
                }
                if (!full) {
                    pf_mask32(s2, 64, lo_rel, hi_rel);
                    pf_mask32(s3, 96, lo_rel, hi_rel);
                }
                const float mx = fmaxf(mx01, pf_max64(s2, s3)) * sl2;  // sl2 > 0: the maximum commutes with the scale
                bool need = false;
                if (t == t0) mref = mx;
                else need = mx > mref + gr.lag;
                // O_g += P_g V(t - 1) has read P and written O (where the scores do not come early, their barrier says that)
                auto products_done = [&]() {
                    if (!C::EARLY || t == t0) return true;
                    const bool done = p3_wait(bar0 + 8 * (C::PV + g), (sc - 1) & 1, abort_flag);
                    tc_fence_after();
                    return done;
                };
                // rows whose maximum moved: O goes to the new reference
                const bool move = __any_sync(0xffffffffu, need);
                float f = 1.0f;
                if (move) {
                    if (need) f = fast_exp2(mref - mx), mref = mx;
                    l *= f;
                    if (!C::EARLY) {
#pragma unroll 1
                        for (int ch = 0; ch < HD / 32; ++ch) {
                            uint32_t o[32];
                            tc_ld32(o_col + 32 * ch, o);
                            tc_wait_ld_for(o);
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[i] = f2u(u2f(o[i]) * f);
                            tc_st32(o_col + 32 * ch, o);
                        }
                    }
                }
                const float ms = mref == -INFINITY ? 0.0f : mref;
                const uint64_t sc2 = pk2(sl2, sl2), nm2 = pk2(-ms, -ms);
                uint64_t acc_a = pk2(0.0f, 0.0f), acc_b = acc_a;
                uint32_t pr[16];
                if (C::TURNS) ok = my_turn();
                if (!ok) break;
                pf_exp32<BF16>(s0, sc2, nm2, acc_a, pr);
                ok = products_done();
                if (!ok) break;
                tc_st16(p_col, pr);
                if (C::EARLY && move) {
                    // The products of the last tile have run under the first exponentials; the row of O comes under the next ones.
                    uint32_t oa[32], ob[32];
                    tc_ld32(o_col, oa);
                    tc_ld32(o_col + 32, ob);
                    pf_exp32<BF16>(s1, sc2, nm2, acc_b, pr);
                    tc_wait_ld_for(oa);
                    tc_wait_ld_for(ob);
#pragma unroll
                    for (int i = 0; i < 32; ++i) oa[i] = f2u(u2f(oa[i]) * f), ob[i] = f2u(u2f(ob[i]) * f);
                    tc_st32(o_col, oa);
                    tc_st32(o_col + 32, ob);
                } else {
                    pf_exp32<BF16>(s1, sc2, nm2, acc_b, pr);
                }
                tc_st16(p_col + 16, pr);
                pf_exp32<BF16>(s2, sc2, nm2, acc_a, pr);
                tc_st16(p_col + 32, pr);
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[C::P0 + g]);
                pf_exp32<BF16>(s3, sc2, nm2, acc_b, pr);
                tc_st16(p_col + 48, pr);
                if (C::TURNS) pass_turn();
                tc_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars[C::P1 + g]);
                ++sc;
                ++tk;
                float a0, a1, b0, b1;
                upk2(acc_a, a0, a1);
                upk2(acc_b, b0, b1);
                l += (a0 + a1) + (b0 + b1);
            }
            if (!ok) break;
            // the next item's figures while the last products run
            const P3Item cur = it;
            const bool any = t1 > t0;
            more = begin(k);
            if (!ok) break;
            if (any) {
                if (!(ok = p3_wait(bar0 + 8 * (C::O + g), oc & 1, abort_flag))) break;
                ++oc;
                tc_fence_after();
            }
            // ---- the row of the output: O / l, or zeros
            const float inv = l > 0.0f ? p.vd / l : 0.0f;
            // 64 elements of the warp's 32 rows at a time through shared memory, so that eight lanes write 128 bytes of a row
            // (a lane that writes its own row leaves every store in 32 lines)
            uint8_t *const stage = smem + C::SM_OUT + warp * 4096;
            if (p.n_splits > 1 || p.o_f32) {
                // f32 rows, 32 elements at a time: outputs, or a key split with the logarithm of the row's sum for fa_combine_kernel
                float *const dst = p.n_splits > 1 ? p.part_o : reinterpret_cast<float *>(p.o);
                const uint64_t part = (uint64_t)cur.split * p.rows_total;
                auto out_row = [&](uint32_t rr) { return (cur.q0 + (rr >> cur.gl)) * p.hq + (cur.hk << cur.gl) + (rr & ((1u << cur.gl) - 1)); };
                const uint32_t r = cur.row0 + g * PF_BM + w4 * 32 + lane;
                if (p.n_splits > 1 && r < cur.R) p.part_lse[part + out_row(r)] = l == 0.0f ? -INFINITY : mref * 0.6931471805599453f + logf(l);  // a NaN stays one
#pragma unroll 1
                for (uint32_t c0 = 0; c0 < p.d; c0 += 32) {
                    uint32_t o[32];
                    if (any) {
                        tc_ld32(o_col + c0, o);
                        tc_wait_ld_for(o);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = 0u;
                    }
#pragma unroll
                    for (int v4 = 0; v4 < 8; ++v4)
                        *reinterpret_cast<float4 *>(stage + lane * 128 + ((v4 ^ (lane & 7)) << 4)) =
                            make_float4(u2f(o[4 * v4]) * inv, u2f(o[4 * v4 + 1]) * inv, u2f(o[4 * v4 + 2]) * inv, u2f(o[4 * v4 + 3]) * inv);
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint32_t row = i * 4 + (lane >> 3), c4 = lane & 7, rr = cur.row0 + g * PF_BM + w4 * 32 + row;
                        const float4 w = *reinterpret_cast<const float4 *>(stage + row * 128 + ((c4 ^ (row & 7)) << 4));
                        if (rr < cur.R && c0 + 4 * c4 < p.d) *reinterpret_cast<float4 *>(dst + (part + out_row(rr)) * p.d + c0 + 4 * c4) = w;
                    }
                    __syncwarp();
                }
                tc_fence_before();
                continue;
            }
#pragma unroll 1
            for (int hf = 0; hf < C::HALVES; ++hf) {
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t o[32];
                    if (any) {
                        tc_ld32(o_col + 64 * hf + 32 * ch, o);
                        tc_wait_ld_for(o);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = 0u;
                    }
#pragma unroll
                    for (int v4 = 0; v4 < 4; ++v4) {
                        uint4 w;
                        w.x = pf_pack2<BF16>(u2f(o[8 * v4]) * inv, u2f(o[8 * v4 + 1]) * inv);
                        w.y = pf_pack2<BF16>(u2f(o[8 * v4 + 2]) * inv, u2f(o[8 * v4 + 3]) * inv);
                        w.z = pf_pack2<BF16>(u2f(o[8 * v4 + 4]) * inv, u2f(o[8 * v4 + 5]) * inv);
                        w.w = pf_pack2<BF16>(u2f(o[8 * v4 + 6]) * inv, u2f(o[8 * v4 + 7]) * inv);
                        *reinterpret_cast<uint4 *>(stage + lane * 128 + (((ch * 4 + v4) ^ (lane & 7)) << 4)) = w;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t row = i * 4 + (lane >> 3), c8 = lane & 7, rr = cur.row0 + g * PF_BM + w4 * 32 + row;
                    const uint4 w = *reinterpret_cast<const uint4 *>(stage + row * 128 + ((c8 ^ (row & 7)) << 4));
                    const uint64_t orow = (cur.q0 + (rr >> cur.gl)) * p.hq + (cur.hk << cur.gl) + (rr & ((1u << cur.gl) - 1));
                    if (rr < cur.R && 64 * hf + 8 * c8 < p.d)
                        *reinterpret_cast<uint4 *>(reinterpret_cast<uint16_t *>(p.o) + orow * p.d + 64 * hf + 8 * c8) = w;
                }
                __syncwarp();
            }
            tc_fence_before();  // O has been read before the next item's first P is announced
        }
        if (!ok) *abort_flag = 1;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == P3_OWNER) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    if (tid == 0 && *abort_flag) atomicExch(&g_wait_failed, 1);
}

// ---- tensor maps -------------------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *,
                                  const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
    static const EncodeTiledFn fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = nullptr;
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    return fn;
}
// What a map says of K or V: a (batch, kv head, key, d) tensor of 16-bit elements with element strides s_b, s_h, s_s and
// contiguous head dim, rank 4: head dim first, the other three in ascending order of stride (entries of extent 1 last).
// `order` gets the places of head, key and batch (two bits each). False when no map can describe the tensor.
struct KvDims {
    uint64_t size[3], stride[3];
    uint32_t order;
};
static bool kv_dims(KvDims *m, const void *base, uint64_t nb, uint64_t hkv, uint64_t lk, uint64_t d_, uint64_t s_b, uint64_t s_h, uint64_t s_s) {
    if (reinterpret_cast<uintptr_t>(base) & 15) return false;
    struct Dim {
        uint64_t size, stride;
        int role;
    } d[3] = {{hkv, s_h * 2, 0}, {lk, s_s * 2, 1}, {nb, s_b * 2, 2}};
    std::stable_sort(d, d + 3, [](const Dim &a, const Dim &c) {
        if ((a.size == 1) != (c.size == 1)) return c.size == 1;  // entries of extent 1 go last
        return a.size > 1 && a.stride < c.stride;
    });
    uint64_t prev = d_ * 2;
    m->order = 0;
    for (int i = 0; i < 3; ++i) {
        if (d[i].size == 0) return false;
        if (d[i].size == 1) {
            d[i].stride = (d_ * 2 + 15) / 16 * 16;  // any legal value: the coordinate is always 0
        } else {
            if ((d[i].stride & 15) || d[i].stride < prev || d[i].stride >= (1ull << 40) || d[i].size > (1ull << 31)) return false;
            prev += d[i].stride * (d[i].size - 1);
        }
        m->size[i] = d[i].size;
        m->stride[i] = d[i].stride;
        m->order |= (uint32_t)i << (2 * d[i].role);
    }
    return true;
}
// boxes of 64 elements x `keys` keys, 128-byte swizzle; elements past the head dim and keys past the end read as zeros
static bool make_kv_map(CUtensorMap *m, const KvDims &k, const void *base, bool bf16, uint64_t d, uint32_t keys) {
    const cuuint64_t dims[4] = {(cuuint64_t)d, k.size[0], k.size[1], k.size[2]};
    const cuuint64_t strides[3] = {k.stride[0], k.stride[1], k.stride[2]};
    cuuint32_t box[4] = {64, 1, 1, 1};
    box[1 + ((k.order >> 2) & 3u)] = keys;
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    const EncodeTiledFn enc = encode_tiled_fn();
    return enc && enc(m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<void *>(base), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The (batch, token, head, d) query tensor as a rank-5 map (element, head in group, kv head, token, batch entry) whose box of
// 64 x G x 1 x 256 / G lands as 256 packed rows (row = token * G + head in group). Sequences of different lengths: one
// batch entry of all tokens.
static bool q_strides(const FaParams &p, cuuint64_t (&strides)[4]) {
    const uint64_t G = p.group, row = (uint64_t)p.d * 2;
    if (G == 0 || G > 256 || (G & (G - 1)) || (reinterpret_cast<uintptr_t>(p.q) & 15)) return false;
    strides[0] = p.q_sh * 2;
    strides[1] = G * p.q_sh * 2;
    strides[2] = p.q_ss * 2;
    strides[3] = p.q_sb * 2;
    if (G == 1) strides[0] = (row + 15) / 16 * 16;
    if (p.hkv == 1) strides[1] = strides[0] * G;
    if (p.varlen || p.b == 1) strides[3] = strides[2];
    if (!p.varlen && p.lq == 1) strides[2] = strides[1];
    for (int i = 0; i < 4; ++i)
        if ((strides[i] & 15) || strides[i] < row || strides[i] >= (1ull << 40)) return false;
    return true;
}
static bool make_q_map(CUtensorMap *m, const FaParams &p, bool bf16) {
    cuuint64_t strides[4];
    if (!q_strides(p, strides)) return false;
    const uint64_t G = p.group;
    const cuuint64_t dims[5] = {(cuuint64_t)p.d, G, p.hkv, p.varlen ? p.rows_total / p.hq : p.lq, p.varlen ? 1u : p.b};
    const cuuint32_t box[5] = {64, (cuuint32_t)G, 1, (cuuint32_t)(P3_ROWS / G), 1};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const EncodeTiledFn enc = encode_tiled_fn();
    return enc && enc(m, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<void *>(p.q), dims, strides, box, estr,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// K and V of a call as maps see them. Sequences of different lengths are one batch entry of keys without an end: the kernel
// copies by tensor map only tiles that lie inside a sequence.
static bool kv_dims_of(const FaParams &p, KvDims *k, KvDims *v) {
    const uint64_t nb = p.varlen ? 1 : p.b, n = p.varlen ? (1ull << 31) : p.lk;
    return kv_dims(k, p.k, nb, p.hkv, n, p.d, p.k_sb, p.k_sh, p.k_ss) && kv_dims(v, p.v, nb, p.hkv, n, p.d, p.v_sb, p.v_sh, p.v_ss);
}

bool fa_kv_maps(const FaParams &p, bool bf16, uint32_t keys, CUtensorMap *tm_k, CUtensorMap *tm_v, uint32_t *order) {
    KvDims k, v;
    if (p.no_maps || !kv_dims_of(p, &k, &v)) return false;
    if (!tm_k) return true;
    *order = k.order | (v.order << 8);
    return make_kv_map(tm_k, k, p.k, bf16, p.d, keys) && make_kv_map(tm_v, v, p.v, bf16, p.d, keys);
}

enum { PF_NONE = 0, PF_ROWS128, PF_ROWS256, PF_TMA };
// More rows than a decode call has (up to 16 rows the keys are read by warps of their own: fa_decode_tma.cu). With 17 to 511 rows
// a block's products run partly on rows that do not exist, and still beat the 64-row tiles of mma.sync: 60 tokens, 32 / 8 heads of
// 128: 26 -> 10 us; 8 x 200 tokens, 16 heads of 128: 65 -> 13; 16 x 400 tokens, 16 heads of 64: 188 -> 41. One item per SM bounds the
// small ones, so few items are split along the keys (fa_plan).
constexpr uint64_t P3_MIN_ROWS = 17;
static int fa_prefill_route(const FaParams &p, bool kv16) {
    if (!kv16 || p.kv_kind != 0) return PF_NONE;
    if (p.q_dtype != B200_F16 && p.q_dtype != B200_BF16) return PF_NONE;
    if (p.softcap > 0.0f || p.alibi != nullptr) return PF_NONE;
    if (!(p.scale * p.kd > 0.0f)) return PF_NONE;  // the row maximum is taken before the scale is applied
    if (reinterpret_cast<uintptr_t>(p.o) & 15) return PF_NONE;  // rows are stored in 16-byte pieces
    static const bool off = [] { const char *e = diag_env("B200_FA_NO_TCGEN05"); return e && *e == '1'; }();
    if (off) return PF_NONE;
    const uint64_t rows = (uint64_t)p.lq * p.group;
    cuuint64_t qs[4];
    static const bool no_tma = [] { const char *e = diag_env("B200_FA_NO_TMA"); return e && *e == '1'; }();
    if (!no_tma && rows >= P3_MIN_ROWS && p.d <= 128 && p.lk < (1u << 31) && rows < (1ull << 31) &&
        (rows + P3_ROWS - 1) / P3_ROWS * p.b * p.hkv < (1ull << 31) && q_strides(p, qs) &&
        fa_kv_maps(p, false, 0, nullptr, nullptr, nullptr))
        return PF_TMA;
    // tensors that no map describes: 16-byte chunks, head dim 128
    if (p.d != PF_D || rows < 4 * PF_BM) return PF_NONE;  // short chunks and decode stay on the mma.sync kernel
    if (p.o_f32) return PF_NONE;  // these two kernels store 16-bit rows only
    if ((reinterpret_cast<uintptr_t>(p.q) & 15) || ((p.q_sb | p.q_ss | p.q_sh) & 7)) return PF_NONE;
    static const long force = [] { const char *e = diag_env("B200_FA_TC_ROWS"); return e ? atol(e) : 0l; }();  // 128 or 256: tile height
    if (force == 128) return PF_ROWS128;
    if (force == 256) return PF_ROWS256;
    // 256-row blocks halve the K / V traffic per product and overlap softmax with products inside the block; they
    // need enough blocks to fill the device
    return rows >= 1024 ? PF_ROWS256 : PF_ROWS128;
}
bool fa_prefill_sm100_supported(const FaParams &p, bool kv16) { return fa_prefill_route(p, kv16) != PF_NONE; }
uint32_t fa_prefill_sm100_splits(const FaParams &p, uint32_t sms) {
    if (p.varlen || fa_prefill_route(p, p.kv_kind == 0) != PF_TMA) return 1;
    // Where the items leave SMs idle: as many key splits as give each SM one, of at least four key tiles (about 8 us; a partial
    // result and the combine grid cost 4)
    // 256 query tokens over 8192 keys, 32 / 8 heads of 128: 145 -> 48 us; 300 over 12 000, 8 / 1 heads: 392 -> 30; 8 tokens x 2 over 4000 keys: 59 -> 24.
    const uint64_t items = ((uint64_t)p.lq * p.group + P3_ROWS - 1) / P3_ROWS * p.b * p.hkv, keys = p.wl >= 0 ? std::min<uint64_t>(p.lk, (uint64_t)p.wl + P3_ROWS) : p.lk;
    return (uint32_t)std::max<uint64_t>(std::min<uint64_t>(std::min<uint64_t>(sms / std::max<uint64_t>(items, 1), keys / (4 * P3_BN)), 64), 1);
}

// shared memory opt-in, once per kernel, thread and device
template <typename K>
static int pf_opt_in(K kern, uint32_t bytes, bool (&done)[16]) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 16 && !done[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return set_error(B200_ERR_LAUNCH, "flash_attn (tcgen05 tiles): shared memory opt-in: %s", cudaGetErrorString(e));
        done[dev] = true;
    }
    return B200_OK;
}

template <int HD, bool BF16>
static int fa_prefill_tma_launch(const FaParams &p, cudaStream_t stream) {
    CUtensorMap tm_k, tm_v, tm_q;
    P3Grid gr;
    if (!fa_kv_maps(p, BF16, P3_BN, &tm_k, &tm_v, &gr.tm_order) || !make_q_map(&tm_q, p, BF16)) return FA_NO_MAP;
    static thread_local bool done[16] = {};
    const int rc = pf_opt_in(fa_prefill_tma_kernel<HD, BF16>, P3<HD>::SMEM, done);
    if (rc) return rc;
    const uint64_t rows = (uint64_t)p.lq * p.group, pair_bytes = std::max<uint64_t>((uint64_t)p.lk * p.d * 4, 1);
    gr.tiles = (uint32_t)((rows + P3_ROWS - 1) / P3_ROWS);
    gr.pairs = p.b * p.hkv;
    gr.hpc = (uint32_t)std::min<uint64_t>(std::max<uint64_t>((64ull << 20) / pair_bytes, 1), gr.pairs);
    gr.items = gr.tiles * gr.pairs * p.n_splits;
    gr.group_log2 = 0;
    while ((1u << gr.group_log2) < p.group) ++gr.group_log2;
    // If a row's reference is its maximum, its largest weight is 1, which 16 bits hold exactly; one that lags makes the error of the
    // output 4 % larger (f16, 1000 keys of 64: 2.78e-4 -> 2.90e-4 against 64 bits). Exact maxima rescale O in most tiles: 8 x 1000
    // tokens, 16 heads of 64: 74.5 -> 79.0 us; heads of 96 in packed prompts: 142 -> 152. So a lag only where rows of O are longest
    // and the calls too, as in the 16-byte chunk tiles that serve such calls where no map describes the tensors.
    gr.lag = p.d == 128 && rows >= 512 && !p.copies ? PF_SLACK : 0.0f;
    fa_prefill_tma_kernel<HD, BF16><<<gr.items, P3_THREADS, P3<HD>::SMEM, stream>>>(p, tm_k, tm_v, tm_q, gr);
    return check_launch("flash_attn (tcgen05 tiles)");
}

int fa_prefill_sm100_launch(const FaParams &p, bool bf16, cudaStream_t stream) {
    const int route = fa_prefill_route(p, p.kv_kind == 0);
    if (route == PF_TMA) {
        if (p.d <= 64) return bf16 ? fa_prefill_tma_launch<64, true>(p, stream) : fa_prefill_tma_launch<64, false>(p, stream);
        return bf16 ? fa_prefill_tma_launch<128, true>(p, stream) : fa_prefill_tma_launch<128, false>(p, stream);
    }
    const uint64_t rows = (uint64_t)p.lq * p.group;
    static thread_local bool done[2][2][16] = {};
    if (route == PF_ROWS256) {
        const int rc = bf16 ? pf_opt_in(fa_prefill_sm100_kernel2<true>, P2_SMEM, done[0][1]) : pf_opt_in(fa_prefill_sm100_kernel2<false>, P2_SMEM, done[0][0]);
        if (rc) return rc;
        const dim3 grid((unsigned)((rows + P2_ROWS - 1) / P2_ROWS), p.hkv, p.b);
        if (bf16) fa_prefill_sm100_kernel2<true><<<grid, P2_THREADS, P2_SMEM, stream>>>(p);
        else fa_prefill_sm100_kernel2<false><<<grid, P2_THREADS, P2_SMEM, stream>>>(p);
    } else {
        const int rc = bf16 ? pf_opt_in(fa_prefill_sm100_kernel<true>, PF_SMEM, done[1][1]) : pf_opt_in(fa_prefill_sm100_kernel<false>, PF_SMEM, done[1][0]);
        if (rc) return rc;
        const dim3 grid((unsigned)((rows + PF_BM - 1) / PF_BM), p.hkv, p.b);
        if (bf16) fa_prefill_sm100_kernel<true><<<grid, PF_THREADS, PF_SMEM, stream>>>(p);
        else fa_prefill_sm100_kernel<false><<<grid, PF_THREADS, PF_SMEM, stream>>>(p);
    }
    return check_launch("flash_attn (tcgen05 tiles)");
}

}  // namespace b200

using namespace b200;

// 1 when a bounded device-side wait of the attention kernels has run out since the library was
// loaded (the call that met it wrote zeros or partial rows); synchronizes the device.
namespace b200 {
int decode_wait_status();  // tq_decode.cu: the same flag of the kernels over packed rows
int decode_wait_clear();
}
extern "C" int b200_device_wait_status(void) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_wait_failed, sizeof(int)) != cudaSuccess) return -1;
    const int d = b200::decode_wait_status(), f = b200::fa_decode_wait_status();
    if (d < 0 || f < 0) return -1;
    return (v != 0 || d != 0 || f != 0) ? 1 : 0;
}

// B200_ERR_DEVICE_WAIT when a bounded device-side wait has run out on the current device since the library was loaded
// (or since the flag was last cleared), B200_OK otherwise; clear != 0 resets the flag, after which the tensor-core
// prefill kernels run again (they return at once, writing nothing, while it is set).
extern "C" int b200_device_wait_check(int clear) {
    const int st = b200_device_wait_status();
    if (st < 0) return set_error(B200_ERR_LAUNCH, "device_wait_check: the flag cannot be read (%s)", cudaGetErrorString(cudaGetLastError()));
    if (clear) {
        const int zero = 0;
        if (cudaMemcpyToSymbol(g_wait_failed, &zero, sizeof(int)) != cudaSuccess || b200::decode_wait_clear() != 0 || b200::fa_decode_wait_clear() != 0)
            return set_error(B200_ERR_LAUNCH, "device_wait_check: the flag cannot be cleared");
    }
    if (st) return set_error(B200_ERR_DEVICE_WAIT, "a bounded device-side wait ran out: the outputs of the call that met it are incomplete");
    return B200_OK;
}
