#define FA_INST_HD 128
#define FA_INST_T __half
#define FA_INST_NAME launch_decode_128_fp16
#define FA_INST_CONFIGS FA_DECODE_CONFIGS_128
#include "decode_inst.inc"
