// Tells a deposit sink the box its next contributions lie in: NX x NY cells
// from (i0, j0).  A sink that wants to know has a member template
// box<NX, NY>(i0, j0); for any other the call does nothing.  Plain C++ (the host
// compiles it with the FP32 deposit's header).
#pragma once

namespace csrst {

template <int NX, int NY, class Sink>
__device__ __forceinline__ auto open_box(Sink &s, int i0, int j0, int)
    -> decltype(s.template box<NX, NY>(i0, j0), void()) {
  s.template box<NX, NY>(i0, j0);
}
template <int NX, int NY, class Sink>
__device__ __forceinline__ void open_box(Sink &, int, int, long) {}

}  // namespace csrst
