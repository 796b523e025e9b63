// FFT passes of some line lengths, single precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<float, 25>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 49>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 63>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 84>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 128>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
