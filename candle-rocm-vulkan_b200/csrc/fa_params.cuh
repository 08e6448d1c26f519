// Parameters shared by the dense attention kernels (fa_dense.cu: mma.sync rows and tiles for every
// shape; fa_prefill_sm100.cu: tcgen05 tiles for long prefill chunks).
#pragma once
#include "common.cuh"

struct CUtensorMap_st;

namespace b200 {

struct FaParams {
    const void *q, *k, *v;
    void *o;
    float *part_o, *part_lse;
    const uint32_t *cu_q, *cu_k;
    const float *alibi;
    uint32_t b, lq, lk, hq, hkv, d, group;
    uint64_t q_sb, q_ss, q_sh, k_sb, k_ss, k_sh, v_sb, v_ss, v_sh;
    float scale, softcap, kd, vd;
    int32_t wl, wr;
    uint32_t alibi_bs, varlen, n_splits;
    int32_t q_dtype;  // dtype of q and o
    int32_t kv_kind;  // 0: 16-bit elements of the mma type, 1: E4M3 bytes, 2: f32
    uint64_t rows_total;  // total_q * hq
    // paged K / V (b200_flash_attn_paged): the blocks, and the keys before every block (n_pages + 1 entries, the last one
    // the total), written by a prefix kernel in front of the attention; null for dense tensors
    const B200Page *pages;
    const uint32_t *pg_keys;
    uint32_t n_pages;
    uint32_t no_maps;  // the driver has refused a tensor map of this call's tensors: kernels that need none
    uint32_t copies;  // q, k and v are 16-bit copies of the call's tensors
    uint32_t o_f32;  // outputs are f32 (over copies); only fa_prefill_tma_kernel writes them
};

// prefill tiles on the 5th generation tensor cores (fa_prefill_sm100.cu)
bool fa_prefill_sm100_supported(const FaParams &p, bool kv16);
uint32_t fa_prefill_sm100_splits(const FaParams &p, uint32_t sms);  // key splits (part_o, part_lse, then fa_combine_kernel)
constexpr int FA_NO_MAP = 1;  // the launches below: nothing was launched, the driver refuses a tensor map
int fa_prefill_sm100_launch(const FaParams &p, bool bf16, cudaStream_t stream);

// Tensor maps of K and V (boxes of 64 elements x `keys` keys, 128-byte swizzle; past the head dim and past the last key zeros
// arrive). `order`: the coordinates' places of head, key and batch entry, two bits each, K in bits 0-5, V in bits 8-13. With
// k == null only whether maps can describe the tensors. fa_prefill_sm100.cu.
bool fa_kv_maps(const FaParams &p, bool bf16, uint32_t keys, CUtensorMap_st *k, CUtensorMap_st *v, uint32_t *order);

// decode over 16-bit K / V by tensor copies (fa_decode_tma.cu): grid (1, hkv, b * n_splits)
bool fa_decode_tma_takes(const FaParams &p, bool paged, uint32_t sms);
int fa_decode_tma_launch(const FaParams &p, bool bf16, dim3 grid, cudaStream_t stream);
int fa_decode_wait_status();
int fa_decode_wait_clear();

}  // namespace b200
