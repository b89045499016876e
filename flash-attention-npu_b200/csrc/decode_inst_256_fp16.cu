#define FA_INST_HD 256
#define FA_INST_T __half
#define FA_INST_NAME launch_decode_256_fp16
#define FA_INST_CONFIGS FA_DECODE_CONFIGS_256
#include "decode_inst.inc"
