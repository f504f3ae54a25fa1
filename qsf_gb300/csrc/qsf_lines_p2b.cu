// 1D step kernels of power-of-two lines, 8192 .. 32768 points.
#include <vector>
#include "qsf_kernels.cuh"
namespace qsf {
void add_lines_p2b(std::vector<LineKernels>& out) {
  out.push_back(make_line<Four<64, 128, 8>>());
  out.push_back(make_line<Four<128, 128, 8, 8>>());
  out.push_back(make_line<Four<128, 256, 8, 8>, false>());  // a convolution length
}
}  // namespace qsf
