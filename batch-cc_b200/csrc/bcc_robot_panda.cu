// bcc_robot_panda.cu -- the checker pipeline instantiated for the Panda robot.
#include "bcc.h"
#include "robot_panda.h"
#include "bcc_pipeline.cuh"

namespace bcc {

__constant__ DevTables<PandaModel> c_tab_panda;
__device__ DevTables<PandaModel> g_tab_panda;  // the same tables for lane-indexed reads

template <>
__device__ __forceinline__ const DevTables<PandaModel>& tab<PandaModel>() {
    return c_tab_panda;
}

template <>
__device__ __forceinline__ const DevTables<PandaModel>& lane_tab<PandaModel>() {
    return g_tab_panda;
}

// Panda's elbow and forearm spheres (links 3 to 6).
template <>
constexpr bool fk_x_first<PandaModel>(int pos) {
    return pos == 4 || pos == 38 || pos == 39 || (pos >= 42 && pos <= 47) || (pos >= 50 && pos <= 52) || pos == 55;
}

static cudaError_t upload_panda_tables() {
    return upload_to<PandaModel>(g_tab_panda, c_tab_panda);
}

extern const RobotOps kPandaOps = robot_ops_of<PandaModel>(BCC_ROBOT_PANDA, upload_panda_tables);

}  // namespace bcc
