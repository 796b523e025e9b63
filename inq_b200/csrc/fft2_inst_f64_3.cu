// FFT passes of some line lengths, double precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<double, 20>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 28>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 36>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 50>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 60>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 84>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 100>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 112>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
