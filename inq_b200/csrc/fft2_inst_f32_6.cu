// FFT passes of some line lengths, single precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<float, 42>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 56>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 81>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 108>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 112>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
