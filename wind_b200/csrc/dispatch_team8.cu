// dispatch_team8.cu -- team kernels with NMAX = 8 (one file per NMAX so
// the instantiations compile in parallel).
#include "api_internal.h"
#include "team_kernel.cuh"

namespace wind {

using TeamFn = void (*)(KParams, int);

TeamFn team_fn_8(int method, int ctrl) {
    if (method == WIND_METHOD_SIE)
        return ctrl == WIND_CTRL_GOLD ? k_team<8, WIND_METHOD_SIE, WIND_CTRL_GOLD>
                                      : k_team<8, WIND_METHOD_SIE, WIND_CTRL_DEVICE>;
    return ctrl == WIND_CTRL_GOLD ? k_team<8, WIND_METHOD_RK2, WIND_CTRL_GOLD>
                                  : k_team<8, WIND_METHOD_RK2, WIND_CTRL_DEVICE>;
}

}  // namespace wind
