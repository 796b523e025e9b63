// FFT passes of some line lengths, single precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<float, 27>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 45>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 70>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 90>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 120>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
