#pragma once
struct __nv_bfloat16 {
  unsigned short bits;
};
float __bfloat162float(__nv_bfloat16);
__nv_bfloat16 __float2bfloat16_rn(float);
