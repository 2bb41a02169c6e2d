// Offsets of the convolution operands on the host: reads lines
//   op B-channels c0 H W m     (op: x, z or w for the forward, data-gradient and
//                               weight-gradient operand; y for the forward result)
// and prints offset, row, column and batch of pixel m.
#include <cinttypes>
#include <cstdio>

#include "conv_ops.cuh"

int main() {
  using namespace gv::cnn;
  char op;
  int C, c0, H, W, m;
  while (std::scanf(" %c %d %d %d %d %d", &op, &C, &c0, &H, &W, &m) == 6) {
    Pixel p{};
    if (op == 'x' || op == 'y') {
      ConvFwdOp o{};
      o.xC = o.yC = C;
      o.xc0 = o.yc0 = c0;
      o.H = H;
      o.W = W;
      p = o.pixel(m);
      if (op == 'y') p.off = o.row(m).off;
    } else if (op == 'z') {
      ConvBwdDataOp o{};
      o.zC = C;
      o.zc0 = c0;
      o.H = H;
      o.W = W;
      p = o.pixel(m);
    } else {
      ConvBwdWeightOp o{};
      o.xC = C;
      o.xc0 = c0;
      o.H = H;
      o.W = W;
      p = o.pixel(m);
    }
    std::printf("%" PRId64 " %d %d %d\n", (int64_t)p.off, p.y, p.x, p.b);
  }
  return 0;
}
