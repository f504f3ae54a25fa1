// 1D step kernels of lines of 3 2^k points, 384 .. 24576.
#include <vector>
#include "qsf_kernels.cuh"
namespace qsf {
void add_lines_r3(std::vector<LineKernels>& out) {
  out.push_back(make_line<Four<16, 24, 1>>());
  out.push_back(make_line<Four<16, 48, 1>>());
  out.push_back(make_line<Four<32, 48, 4>>());
  out.push_back(make_line<Four<32, 96, 8>>());
  out.push_back(make_line<Four<64, 96, 8>>());
  out.push_back(make_line<Four<64, 192, 8>>());
  out.push_back(make_line<Four<128, 192, 8, 8>, false>());  // a convolution length
}
}  // namespace qsf
