// Which kernel serves a call of the tensor-core forward (fp16 storage, head_dim 8 or 16).
#include "attn_kernels.cuh"
#include "attn_tc.cuh"

namespace s3d {

// Head mode of the tensor-core kernels for a call (see attn_tc.cuh).
int attn_tc_head_mode(const AttnArgs &a)
{
    if (a.hd == 8) return tc::HDM_PAIR8;
    return (a.H & 1) ? tc::HDM_SINGLE16 : tc::HDM_PAIR16;
}

bool attn_tc_supported(const AttnArgs &a)
{
    if (a.meta.R + a.meta.D - 1 > 384) return false;         // larger tables: the generic path
    if (a.hd == 16 && attn_tc_head_mode(a) == tc::HDM_PAIR16) return attn_tc_fwd_pair16_supported(a);
    return attn_tc_fwd_small_supported(a);
}

int attn_tc_forward(const AttnArgs &a, cudaStream_t st)
{
    if (a.W == 0) return S3D_OK;
    return attn_tc_head_mode(a) == tc::HDM_PAIR16 ? attn_tc_forward_pair16(a, st) : attn_tc_forward_small(a, st);
}

}  // namespace s3d
