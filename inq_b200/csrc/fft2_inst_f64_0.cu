// FFT passes of some line lengths, double precision (spread over files for parallel builds).
#include "fft2.cuh"

namespace inqb {
namespace v2 {
template void launch_n<double, 21>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 27>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 35>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 54>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 56>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 80>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 90>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
template void launch_n<double, 128>(Ctx &, const Basis &, const PassArgs<double> &, Geom2, int);
}  // namespace v2
}  // namespace inqb
