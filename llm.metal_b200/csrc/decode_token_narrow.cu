// The whole-token kernel with half of the consumer threads, for layers of little weight (b200_token_plan chooses).
#define B200_TOKEN_NARROW
#include "decode_token_core.cuh"

int b200_tk_launch_narrow(const b200_token_args &a, cudaStream_t st)
{
    void (*kern)(const b200_token_args) =
        a.wtype == B200_WT_Q8 ? (a.d_trace ? decode_token_kernel<B200_WT_Q8, true, false> : decode_token_kernel<B200_WT_Q8, false, false>)
                              : (a.d_trace ? decode_token_kernel<B200_WT_F16, true, false> : decode_token_kernel<B200_WT_F16, false, false>);
    return launch_token(kern, a, st);
}
