// Element-wise kernels of nn.cu that the launch sequences of fno.cpp use and
// the C interface does not carry.
#pragma once

namespace csrst {

// dx = dy GELU'(pre) (pre NULL: dx = dy) of [rows][cols], rows and cols multiples of 64, 16-byte
// aligned pointers: FP32 (dx32, may be NULL), BF16 and the BF16 transpose [cols][rows].
int nn_backward_rows(const float *dy, const float *pre, float *dx32, void *dx16, void *dxT16, int rows, int cols,
                     void *stream);

}  // namespace csrst
