// Stand-in for the bfloat16 header (see cuda_runtime.h beside it).
#pragma once
#include "cuda_runtime.h"
struct __nv_bfloat16 { uint16_t bits; };
inline float __bfloat162float(__nv_bfloat16 v) { return emu_bits<float>((uint32_t)v.bits << 16); }
