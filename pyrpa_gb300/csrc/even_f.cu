// Even-model stages in FP32, and the conversions between bulk types.
#include "even_impl.cuh"

namespace pgb {
PGB_EVEN_INST(float)
template void convert_even<float, double>(const Even&, cx<float>*, const cx<double>*, long long);
template void convert_even<float, dfl>(const Even&, cx<float>*, const cx<dfl>*, long long);
template void convert_even<double, float>(const Even&, cx<double>*, const cx<float>*, long long);
template void convert_even<double, dfl>(const Even&, cx<double>*, const cx<dfl>*, long long);
template void convert_even<dfl, float>(const Even&, cx<dfl>*, const cx<float>*, long long);
template void convert_even<dfl, double>(const Even&, cx<dfl>*, const cx<double>*, long long);
}  // namespace pgb
