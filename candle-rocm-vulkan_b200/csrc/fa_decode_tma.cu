// Decoding attention over dense 16-bit K / V, tiles by tensor copies: the calls of b200_flash_attn whose packed query rows
// (tokens x heads of the group) fit one group of 16, head dims up to 128, tensors that a tensor map describes, and those of b200_flash_attn_paged over such rows (PAGED: the same tiles and the
// same arithmetic, so the same bits; a warp finds its keys in the block table and copies them by 16-byte chunks). The other
// forms (E4M3 or f32 keys, packed sequences, larger heads) stay on fa_dense_kernel.
//
// Bound by memory: every key and value is read once. So nothing stands between a warp and its next tiles: each of the four
// warps of a block streams every fourth tile (16 keys at head dim 128, 32 at 64: 8 KB) through a ring of its own of three
// stages, which its lane 0 refills with tensor copies as soon as the warp has read a stage; no block barrier and no address
// arithmetic in the loop. Two blocks per SM keep 192 KB on their way. S = Q K^T and O += P V run on
// mma.sync m16n8k16 as in fa_dense_kernel, the sums of O are only rescaled in tiles in which a row's maximum moves, and keys
// are only masked where some row needs it. The warps' partial results meet in shared memory at the end, those of the key
// splits in fa_combine_kernel.
//
// Measured against the block-wide double buffer of fa_dense_kernel (us, graph replay, both with their combine grid; B, keys, query /
// kv heads, head dim): 64, 4096, 32 / 8, 128: 224 -> 186 (5.8 TB/s); 64, 4000, 16 / 16, 64: 246 -> 165 (6.3 TB/s); 4, 8000, 8 / 1, 128:
// 60 -> 15; 1, 2000, 16 / 4, 128: 25 -> 11; 1, 200, 32 / 8, 64: 8.8 -> 6.2. The short ones owe most to fa_combine_kernel, whose lanes
// walked the splits one dependent load at a time.
//
// Every wait is bounded; one that runs out raises the flag that b200_device_wait_status reads.
#include <algorithm>
#include <cuda.h>

#include "common.cuh"
#include "fa_params.cuh"

namespace b200 {

constexpr int FD_WARPS = 4, FD_RING = 24576;
constexpr float FD_LOG2E = 1.4426950408889634f, FD_LN2 = 0.6931471805599453f;

__device__ int g_decode_wait_failed = 0;

template <int HD>
struct FD {
    static constexpr int HALVES = HD / 64, KEYS = HD == 64 ? 32 : 16;  // keys per tile: a stage has 8 KB
    static constexpr uint32_t HALF = KEYS * 128, TILE = HALVES * HALF, STAGE = 2 * TILE;  // [K, V][half][key][128 bytes, swizzled]
    static constexpr int NS = FD_RING / STAGE;
    static constexpr int QROW = HD * 2 + 16;  // padded row bytes of Q
    static constexpr uint32_t SM_Q = FD_WARPS * FD_RING, SM_BAR = SM_Q + 16 * QROW, SMEM = SM_BAR + FD_WARPS * NS * 8;
    static_assert(FD_WARPS * 16 * (HD + 2) * 4 <= FD_WARPS * FD_RING, "the merge reuses the rings");
};

__device__ __forceinline__ void fd_ldsm(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void fd_ldsm_trans(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
template <bool BF16>
__device__ __forceinline__ void fd_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if (BF16)
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                     : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                     : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool BF16>
__device__ __forceinline__ uint32_t fd_pack2(float lo, float hi) {
    uint32_t d;
    if (BF16) asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    else asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}
__device__ __forceinline__ void fd_copy(uint32_t dst, const CUtensorMap *map, int c0, int c1, int c2, int c3, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
                 : "memory");
}

template <int HD, bool BF16, bool PAGED>
__global__ void __launch_bounds__(FD_WARPS * 32, 2) fa_decode_tma_kernel(const FaParams p, const __grid_constant__ CUtensorMap tm_k,
                                                                         const __grid_constant__ CUtensorMap tm_v, const uint32_t tm_order) {
    using C = FD<HD>;
    constexpr int KSTEPS = HD / 16, NT = HD / 8, KEYS = C::KEYS, KG = KEYS / 16;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, c = lane & 3;
    const uint32_t ring = smem_u32(smem) + warp * FD_RING, sQ = smem_u32(smem) + C::SM_Q;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + C::SM_BAR) + warp * C::NS;
    const uint32_t D = p.d, hk = blockIdx.y, b = blockIdx.z / p.n_splits, split = blockIdx.z % p.n_splits, G = p.group;
    const int lq = (int)p.lq, lk = PAGED ? (int)min(p.lk, p.pg_keys[p.n_pages]) : (int)p.lk, R = lq * (int)G;
    if (p.n_splits > 1) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // the combine grid may get ready

    // the keys that row r sees
    auto range_of = [&](int r, int &lo, int &hi) {
        const int pos = r / (int)G + lk - lq;
        lo = p.wl >= 0 && pos > p.wl ? min(pos - p.wl, lk) : 0;
        hi = p.wr >= 0 && pos < lk - p.wr - 1 ? pos + p.wr + 1 : lk;
        hi = max(hi, lo);
    };
    int t_lo, t_hi, x0, x1;
    range_of(0, t_lo, x0);
    range_of(R - 1, x1, t_hi);
    t_hi = max(t_hi, t_lo);
    // this split's share, in whole tiles; the warp's tiles are every fourth of them
    const int all = (t_hi - t_lo + KEYS - 1) / KEYS, per = (all + (int)p.n_splits - 1) / (int)p.n_splits;
    const int first = min((int)split * per, all), last = min(first + per, all);
    const int nt = last - first > warp ? (last - first - warp + FD_WARPS - 1) / FD_WARPS : 0;
    auto key_of = [&](int t) { return t_lo + (first + t * FD_WARPS + warp) * KEYS; };
    auto request = [&](int t) {  // lane 0
        const uint32_t st = t % C::NS, dst = ring + st * C::STAGE, bar = smem_u32(&bars[st]);
        const int j = key_of(t);
        mbar_expect_tx(&bars[st], C::STAGE);
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
            const uint32_t ord = kv ? tm_order >> 8 : tm_order, ph = ord & 3u, pk = (ord >> 2) & 3u;
            const int c1 = ph == 0 ? (int)hk : (pk == 0 ? j : (int)b), c2 = ph == 1 ? (int)hk : (pk == 1 ? j : (int)b), c3 = ph == 2 ? (int)hk : (pk == 2 ? j : (int)b);
#pragma unroll
            for (int hf = 0; hf < C::HALVES; ++hf) fd_copy(dst + kv * C::TILE + hf * C::HALF, kv ? &tm_v : &tm_k, 64 * hf, c1, c2, c3, bar);
        }
    };
    // PAGED, all lanes: lane i finds the row of key i in the block table (block n holds the keys pg_keys[n] .. pg_keys[n + 1] - 1 at
    // rows 0 .. of its slab; `page` is at or before the lane's next key), then HD / 8 lanes copy a row
    uint32_t page = 0;
    auto request_paged = [&](int t) {
        const uint32_t dst = ring + (t % C::NS) * C::STAGE;
        const int j = key_of(t) + lane;
        const char *kr = nullptr, *vr = nullptr;
        if (lane < KEYS && j < t_hi) {
            while (page + 1 < p.n_pages && (int)p.pg_keys[page + 1] <= j) ++page;
            const B200Page pd = p.pages[page];
            const uint64_t row = (uint64_t)(j - (int)p.pg_keys[page]), slab = (uint64_t)b * p.hkv + hk;
            kr = reinterpret_cast<const char *>(pd.k) + (slab * pd.k_cap + row) * p.k_ss * 2;
            vr = reinterpret_cast<const char *>(pd.v) + (slab * pd.v_cap + row) * p.v_ss * 2;
        }
        constexpr int LPR = HD / 8;  // lanes per row
        const uint32_t ch = lane % LPR;
#pragma unroll
        for (int i = 0; i < KEYS * LPR / 32; ++i) {
            const int row = i * (32 / LPR) + lane / LPR;
            const char *k_src = reinterpret_cast<const char *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(kr), row));
            const char *v_src = reinterpret_cast<const char *>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(vr), row));
            const bool in = k_src != nullptr && ch * 8 < D;
            const uint32_t at = dst + (ch >> 3) * C::HALF + row * 128 + (((ch & 7) ^ (row & 7)) << 4);
            const void *none = p.pg_keys;  // what is not copied reads as zeros; a source is 16-byte aligned even then, and q need not be
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(in ? k_src + ch * 16 : none), "r"(in ? 16 : 0) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + C::TILE), "l"(in ? v_src + ch * 16 : none), "r"(in ? 16 : 0) : "memory");
        }
    };
    if (PAGED) {
        // the block of the warp's first key: binary search over the prefix sums
        uint32_t lo = 0, hi = p.n_pages;
        while (nt > 0 && lo + 1 < hi) {
            const uint32_t mid = (lo + hi) / 2;
            if ((int)p.pg_keys[mid] <= key_of(0)) lo = mid;
            else hi = mid;
        }
        page = lo;
        for (int t = 0; t < C::NS; ++t) {
            if (t < nt) request_paged(t);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    } else if (lane == 0) {
        for (int i = 0; i < C::NS; ++i) mbar_init(&bars[i], 1);
        mbar_fence_init();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (int t = 0; t < min(nt, C::NS); ++t) request(t);
    }
    // Q -> shared memory (any alignment), then A fragments in registers
    const char *qb = reinterpret_cast<const char *>(p.q);
    for (int idx = tid; idx < 16 * HD; idx += FD_WARPS * 32) {
        const int rr = idx / HD, dd = idx % HD;
        uint16_t v = 0;
        if (rr < R && dd < (int)D) {
            const uint64_t off = b * p.q_sb + (uint64_t)(rr / (int)G) * p.q_ss + (hk * G + rr % (int)G) * p.q_sh + dd;
            if (p.q_dtype == B200_F32) {
                const float f = reinterpret_cast<const float *>(qb)[off];
                v = BF16 ? f_to_bf16_bits(f) : f_to_f16_bits(f);
            } else {
                v = reinterpret_cast<const uint16_t *>(qb)[off];
            }
        }
        *reinterpret_cast<uint16_t *>(smem + C::SM_Q + rr * C::QROW + dd * 2) = v;
    }
    __syncthreads();
    uint32_t qa[KSTEPS][4];
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks) fd_ldsm(sQ + (lane & 15) * C::QROW + (lane >> 4) * 16 + ks * 32, qa[ks][0], qa[ks][1], qa[ks][2], qa[ks][3]);

    // rows g and g + 8 of this lane; rows that do not exist see every key and are never stored
    int r_lo[2] = {0, 0}, r_hi[2] = {lk, lk}, r_pos[2] = {0, 0}, lomax = 0, himin = lk;
    float slope[2] = {0.0f, 0.0f};
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int r = g + 8 * e;
        if (r < R) {
            range_of(r, r_lo[e], r_hi[e]);
            r_pos[e] = r / (int)G + lk - lq;
            if (p.alibi) slope[e] = p.alibi[(size_t)b * p.alibi_bs + hk * G + r % (int)G];
        }
    }
    range_of(R - 1, lomax, x0);
    range_of(0, x0, himin);
    himin = min(himin, t_hi);
    const float sc = p.scale * p.kd, sc2 = sc * FD_LOG2E;
    const bool plain = p.softcap <= 0.0f && p.alibi == nullptr;

    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};  // maxima in units of log 2
    float oacc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n) oacc[n][0] = oacc[n][1] = oacc[n][2] = oacc[n][3] = 0.0f;
    const uint32_t sw = lane & 7;  // the row of a core matrix that the lane addresses: the swizzle's part of it
    bool ok = true;
    for (int t = 0; t < nt; ++t) {
        const uint32_t st = t % C::NS;
        if (PAGED) {
            asm volatile("cp.async.wait_group %0;" ::"n"(C::NS - 1) : "memory");
            __syncwarp();
        } else {
            ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bars[st], (t / C::NS) & 1));
            if (!ok) break;
        }
        const uint32_t tk = ring + st * C::STAGE, tv = tk + C::TILE;
        const int j0 = key_of(t);
        float s[2 * KG][4];
#pragma unroll
        for (int n = 0; n < 2 * KG; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.0f;
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
#pragma unroll
            for (int np = 0; np < KG; ++np) {
                uint32_t b0, b1, b2, b3;
                const uint32_t ch = ks * 2 + ((lane >> 3) & 1);
                fd_ldsm(tk + (ch >> 3) * C::HALF + (np * 16 + (lane & 7) + ((lane >> 4) << 3)) * 128 + (((ch & 7) ^ sw) << 4), b0, b1, b2, b3);
                fd_mma<BF16>(s[2 * np], qa[ks], b0, b1);
                fd_mma<BF16>(s[2 * np + 1], qa[ks], b2, b3);
            }
        }
        const bool full = plain && j0 >= lomax && j0 + KEYS <= himin;
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int n = 0; n < 2 * KG; ++n) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int e = i >> 1;
                float x = s[n][i] * sc2;
                if (!full) {
                    const int j = j0 + 8 * n + 2 * c + (i & 1);
                    if (!plain && (e == 0 || R > 8)) {  // (rows 8 to 15 of a call that has none need no soft cap)
                        x = s[n][i] * sc;
                        if (p.softcap > 0.0f) x = p.softcap * tanhf(x / p.softcap);
                        if (slope[e] != 0.0f) x -= slope[e] * fabsf((float)(r_pos[e] - j));
                        x *= FD_LOG2E;
                    }
                    if (!(j >= r_lo[e] && j < r_hi[e])) x = -INFINITY;
                }
                s[n][i] = x;
                mx[e] = fmaxf(mx[e], x);
            }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 1));
            mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 2));
        }
        if (__any_sync(0xffffffffu, mx[0] > m[0] || mx[1] > m[1])) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float mn = fmaxf(m[e], mx[e]), f = m[e] == -INFINITY ? 0.0f : fast_exp2(m[e] - mn);
                m[e] = mn;
                l[e] *= f;
#pragma unroll
                for (int n = 0; n < NT; ++n) oacc[n][2 * e] *= f, oacc[n][2 * e + 1] *= f;
            }
        }
        const float ms0 = m[0] == -INFINITY ? 0.0f : m[0], ms1 = m[1] == -INFINITY ? 0.0f : m[1];
        uint32_t pa[KG][4];
#pragma unroll
        for (int n = 0; n < 2 * KG; ++n) {
            const float p0 = fast_exp2(s[n][0] - ms0), p1 = fast_exp2(s[n][1] - ms0), p2 = fast_exp2(s[n][2] - ms1), p3 = fast_exp2(s[n][3] - ms1);
            l[0] += p0 + p1;
            l[1] += p2 + p3;
            pa[n >> 1][(n & 1) * 2] = fd_pack2<BF16>(p0, p1);
            pa[n >> 1][(n & 1) * 2 + 1] = fd_pack2<BF16>(p2, p3);
        }
#pragma unroll
        for (int kk = 0; kk < KG; ++kk) {
#pragma unroll
            for (int np = 0; np < NT / 2; ++np) {
                uint32_t b0, b1, b2, b3;
                const uint32_t ch = np * 2 + (lane >> 4);
                fd_ldsm_trans(tv + (ch >> 3) * C::HALF + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * 128 + (((ch & 7) ^ sw) << 4), b0, b1, b2, b3);
                fd_mma<BF16>(oacc[2 * np], pa[kk], b0, b1);
                fd_mma<BF16>(oacc[2 * np + 1], pa[kk], b2, b3);
            }
        }
        __syncwarp();  // the stage has been read
        if (PAGED) {
            if (t + C::NS < nt) request_paged(t + C::NS);
            asm volatile("cp.async.commit_group;" ::: "memory");
        } else if (lane == 0 && t + C::NS < nt) {
            request(t + C::NS);
        }
    }
    if (PAGED) asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!ok) {
        // copies still in flight must land before the block may leave (bounded)
        if (lane == 0)
            for (int i = 0; i < C::NS; ++i) mbar_wait_bounded(&bars[i], 0, 1u << 12), mbar_wait_bounded(&bars[i], 1, 1u << 12);
        atomicExch(&g_decode_wait_failed, 1);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 1);
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 2);
    }
    // the four warps' partial results: [warp][row][HD sums, maximum, sum of weights] over the rings, eight threads per row
    constexpr int MS = HD + 2;
    float *mg = reinterpret_cast<float *>(smem);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        float *dst = mg + (warp * 16 + g + 8 * e) * MS;
#pragma unroll
        for (int n = 0; n < NT; ++n) *reinterpret_cast<float2 *>(dst + 8 * n + 2 * c) = make_float2(oacc[n][2 * e], oacc[n][2 * e + 1]);
        if (c == 0) dst[HD] = m[e], dst[HD + 1] = l[e];
    }
    __syncthreads();
    const int row = tid >> 3, ch = tid & 7;
    if (row >= R) return;
    float f[FD_WARPS], M = -INFINITY, L = 0.0f;
#pragma unroll
    for (int w = 0; w < FD_WARPS; ++w) M = fmaxf(M, mg[(w * 16 + row) * MS + HD]);
    const float ms = M == -INFINITY ? 0.0f : M;
#pragma unroll
    for (int w = 0; w < FD_WARPS; ++w) {
        f[w] = fast_exp2(mg[(w * 16 + row) * MS + HD] - ms);
        L += f[w] * mg[(w * 16 + row) * MS + HD + 1];
    }
    const float inv = L > 0.0f ? p.vd / L : 0.0f;
    const uint64_t orow = ((uint64_t)b * p.lq + row / (int)G) * p.hq + hk * G + row % (int)G, prow = (uint64_t)split * p.rows_total + orow;
#pragma unroll 4
    for (uint32_t dd = 2 * ch; dd < D; dd += 16) {
        float o0 = 0.0f, o1 = 0.0f;
#pragma unroll
        for (int w = 0; w < FD_WARPS; ++w) {
            const float2 v = *reinterpret_cast<const float2 *>(mg + (w * 16 + row) * MS + dd);
            o0 = fmaf(f[w], v.x, o0);
            o1 = fmaf(f[w], v.y, o1);
        }
        if (p.n_splits == 1) {
            store_elem_rt(p.o, orow * D + dd, o0 * inv, p.q_dtype);
            store_elem_rt(p.o, orow * D + dd + 1, o1 * inv, p.q_dtype);
        } else {
            *reinterpret_cast<float2 *>(p.part_o + prow * D + dd) = make_float2(o0 * inv, o1 * inv);
        }
    }
    if (p.n_splits > 1 && ch == 0) p.part_lse[prow] = L == 0.0f ? -INFINITY : M * FD_LN2 + logf(L);  // a NaN stays one
}

bool fa_decode_tma_takes(const FaParams &p, bool paged, uint32_t sms) {
    const uint64_t rows = (uint64_t)p.lq * p.group, blocks = (uint64_t)p.b * p.hkv;
    const uint64_t keys = p.wl >= 0 ? std::min<uint64_t>(p.lk, (uint64_t)p.wl + p.lq) : p.lk;
    // A soft cap costs more than the copies: where the tiles of 32 keys leave a warp more of a few keys than its share, the general
    // kernel's four warps of 16 keys are ahead (us, there and here: up to eight rows, 20 keys 6.3, 6.7; 9 to 16 rows, 11 keys 8.3, 9.7;
    // 132 keys 11.3, 12.4; eight rows, 126 keys 9.5, 8.5).
    if ((p.softcap > 0.0f || p.alibi) && p.d <= 64 && keys <= (rows > 8 ? 192u : 64u)) return false;
    // The general kernel has four blocks per SM up to head dim 64 and three up to 128, this one two. Calls over few keys that are one
    // wave there and two here are ahead there (us, there and here: 432 blocks, 1 row, 58 keys of 64: 6.5, 9.2; 384 blocks, 4 rows,
    // 108 keys 8.6, 10.4, but 468 blocks, 2 rows, 252 keys 13.5, 12.1; 16 rows: 327 blocks, 558 keys of 64 20.1, 22.1; 416 blocks,
    // 34 keys of 128 16.6, 19.9; 390 blocks, 428 keys of 96 27.4, 32.0; 8 rows: 440 blocks, 52 keys of 96 11.5, 15.4; 432 blocks, 384 keys of 128 24.4, 26.4;
    // 336 blocks, 665 keys 39.7, 42.0; 4 rows, 424 blocks, 681 keys of 96: equal).
    if (blocks > 2ull * sms && blocks <= (p.d <= 64 ? 4ull : 3ull) * sms && keys <= (rows <= 8 && p.d <= 64 ? 192u : 704u)) return false;
    return p.kv_kind == 0 && !p.varlen && p.d <= 128 && p.lk > 0 && p.lk < (1u << 31) && (uint64_t)p.lq * p.group <= 16 &&
           (paged || fa_kv_maps(p, false, 0, nullptr, nullptr, nullptr));
}

template <int HD, bool BF16, bool PAGED>
static int launch(const FaParams &p, dim3 grid, cudaStream_t stream) {
    CUtensorMap tm_k, tm_v;
    uint32_t order = 0;
    if (PAGED) memset(&tm_k, 0, sizeof(tm_k)), memset(&tm_v, 0, sizeof(tm_v));
    else if (!fa_kv_maps(p, BF16, FD<HD>::KEYS, &tm_k, &tm_v, &order)) return FA_NO_MAP;
    static thread_local bool done[16] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 16 && !done[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(fa_decode_tma_kernel<HD, BF16, PAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FD<HD>::SMEM);
        if (e != cudaSuccess) return set_error(B200_ERR_LAUNCH, "flash_attn (decode): shared memory opt-in: %s", cudaGetErrorString(e));
        done[dev] = true;
    }
    fa_decode_tma_kernel<HD, BF16, PAGED><<<grid, FD_WARPS * 32, FD<HD>::SMEM, stream>>>(p, tm_k, tm_v, order);
    return check_launch("flash_attn (decode)");
}
int fa_decode_tma_launch(const FaParams &p, bool bf16, dim3 grid, cudaStream_t stream) {
    if (p.pages) {
        if (p.d <= 64) return bf16 ? launch<64, true, true>(p, grid, stream) : launch<64, false, true>(p, grid, stream);
        return bf16 ? launch<128, true, true>(p, grid, stream) : launch<128, false, true>(p, grid, stream);
    }
    if (p.d <= 64) return bf16 ? launch<64, true, false>(p, grid, stream) : launch<64, false, false>(p, grid, stream);
    return bf16 ? launch<128, true, false>(p, grid, stream) : launch<128, false, false>(p, grid, stream);
}

int fa_decode_wait_status() {
    int v = 0;
    return cudaMemcpyFromSymbol(&v, g_decode_wait_failed, sizeof(int)) == cudaSuccess ? v : -1;
}
int fa_decode_wait_clear() {
    const int zero = 0;
    return cudaMemcpyToSymbol(g_decode_wait_failed, &zero, sizeof(int)) == cudaSuccess ? 0 : -1;
}

}  // namespace b200
