// Launch description of an fp32 contraction by tiled copies (tile32.cu), made by the plan compiler.
#pragma once

namespace b200 {
struct Tile32Launch {
  int mode = 0;                              // 0: not used, else how A is fetched (tile32.cu): 1 convolution, 2 rows of k, 3 rows of m
  int M = 0, N = 0, K = 0, G = 1;
  int bn = 64, split = 1;                    // tile width, K split
  // A as a tensor of rank 4, contiguous dimension first (elements), and the box of one copy
  long long dims[4] = {1, 1, 1, 1}, strides[3] = {0, 0, 0};
  unsigned box[4] = {1, 1, 1, 1};
  int ow = 1, oh = 1, kw = 1;                // convolutions: output image, filter width
  int pad_h = 0, pad_w = 0, dil_h = 1, dil_w = 1, cin = 0;
  int c_vec = 0;                             // consecutive n are consecutive floats in C (2: and rows start on 16 bytes)
  long long image_floats() const {           // B split into its two parts, in the order the tiles are used
    return 2ll * G * ((N + bn - 1) / bn) * bn * ((K + 31) / 32) * 32;
  }
};
}  // namespace b200
