// The whole-token kernel with half of the consumer threads, for layers of little weight (b200_token_plan chooses).
#define B200_TOKEN_NARROW
#include "decode_token.cu"
