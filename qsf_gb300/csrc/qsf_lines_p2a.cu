// 1D step kernels of power-of-two lines, 256 .. 4096 points.
#include <vector>
#include "qsf_kernels.cuh"
namespace qsf {
void add_lines_p2a(std::vector<LineKernels>& out) {
  out.push_back(make_line<Four<16, 16, 1>>());
  out.push_back(make_line<Four<16, 32, 1>>());
  out.push_back(make_line<Four<32, 32, 2>>());
  out.push_back(make_line<Four<32, 64, 4>>());
  out.push_back(make_line<Four<64, 64, 8>>());
}
}  // namespace qsf
