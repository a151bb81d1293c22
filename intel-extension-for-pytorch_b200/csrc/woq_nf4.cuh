// The NF4 table: code -> value (reference: csrc/cpu/aten/utils/woq_utils.h:34-51).  A list, not an object: a
// __constant__ variable anywhere in a module costs each of its kernels' launches about 0.7 us, so only the general
// kernel has one and the CTA-pair kernel takes the values as a parameter.
#pragma once

#define WOQ_NF4_VALUES                                                                              \
  {                                                                                                 \
    -1.0f, -0.6961928009986877f, -0.5250730514526367f, -0.39491748809814453f, -0.28444138169288635f, \
        -0.18477343022823334f, -0.09105003625154495f, 0.0f, 0.07958029955625534f,                   \
        0.16093020141124725f, 0.24611230194568634f, 0.33791524171829224f, 0.44070982933044434f,     \
        0.5626170039176941f, 0.7229568362236023f, 1.0f                                              \
  }
