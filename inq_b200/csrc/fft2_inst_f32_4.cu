// FFT passes of some line lengths, single precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<float, 20>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 36>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 54>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 72>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 80>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
template void launch_n<float, 100>(Ctx &, const Basis &, const PassArgs<float> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
