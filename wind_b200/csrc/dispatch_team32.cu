// dispatch_team32.cu -- team kernels with NMAX = 32 (one file per NMAX so
// the instantiations compile in parallel).
#include "api_internal.h"
#include "team_kernel.cuh"

namespace wind {

using TeamFn = void (*)(KParams, int);

TeamFn team_fn_32(int method, int ctrl) {
    if (method == WIND_METHOD_SIE)
        return ctrl == WIND_CTRL_GOLD ? k_team<32, WIND_METHOD_SIE, WIND_CTRL_GOLD>
                                      : k_team<32, WIND_METHOD_SIE, WIND_CTRL_DEVICE>;
    return ctrl == WIND_CTRL_GOLD ? k_team<32, WIND_METHOD_RK2, WIND_CTRL_GOLD>
                                  : k_team<32, WIND_METHOD_RK2, WIND_CTRL_DEVICE>;
}

}  // namespace wind
