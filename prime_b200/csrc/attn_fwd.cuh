// Parameters of the two forward attention kernels (attn_fwd_sm100.cu, attn_fwd128_sm100.cu).
#pragma once
#include "common.cuh"

namespace pb {

struct AttnFwdParams {
    int M, H, KV;
    int hd;             // columns of a head, <= HD
    const int* seq_start;
    __nv_bfloat16* O;
    long long o_stride;
    float* lse2;
    float scale_log2;   // softmax scale * log2(e)
    int* status;
};

int launch_attn_fwd128(const CUtensorMap& tm, const AttnFwdParams& p, cudaStream_t st);
int sm_count();

}  // namespace pb
