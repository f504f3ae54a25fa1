// 1D step kernels of lines held by one CTA as one line.
#include <vector>
#include "qsf_kernels.cuh"
namespace qsf {
void add_lines_one(std::vector<LineKernels>& out) {
  out.push_back(make_line<One<8>>());
  out.push_back(make_line<One<12>>());
  out.push_back(make_line<One<16>>());
  out.push_back(make_line<One<20>>());
  out.push_back(make_line<One<24>>());
  out.push_back(make_line<One<32>>());
  out.push_back(make_line<One<40>>());
  out.push_back(make_line<One<48>>());
  out.push_back(make_line<One<64>>());
  out.push_back(make_line<One<80>>());
  out.push_back(make_line<One<96>>());
  out.push_back(make_line<One<128>>());
  out.push_back(make_line<One<160>>());
  out.push_back(make_line<One<192>>());
  out.push_back(make_line<One<320>>());
}
}  // namespace qsf
