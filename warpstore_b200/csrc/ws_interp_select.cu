// Interpreter instantiations (prefix wsi) of the selection pass.  The scan kernels are
// split over several translation units so that they compile in parallel.
#include "ws_internal.h"
#include "ws_interp.cuh"

WS_K_SELECT(ws::InterpEv, wsi)

namespace ws {
void interpSyms_select(const void** s) {
  s[K_SELECT] = (const void*)wsi_select;
}
}  // namespace ws
