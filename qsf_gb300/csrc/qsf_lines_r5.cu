// 1D step kernels of lines of 5 2^k points, 640 .. 20480.
#include <vector>
#include "qsf_kernels.cuh"
namespace qsf {
void add_lines_r5(std::vector<LineKernels>& out) {
  out.push_back(make_line<Four<16, 40, 1>>());
  out.push_back(make_line<Four<16, 80, 2>>());
  out.push_back(make_line<Four<32, 80, 4>>());
  out.push_back(make_line<Four<64, 80, 8>>());
  out.push_back(make_line<Four<64, 160, 8>>());
  out.push_back(make_line<Four<128, 160, 8, 8>, false>());  // a convolution length
}
}  // namespace qsf
