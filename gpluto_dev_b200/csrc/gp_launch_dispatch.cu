// gp_launch_dispatch.cu -- joins the per-physics launch units of
// gp_launch.cu (compiled once per form and physics, GP_MIXED x GP_PART).
#include "gp_kernels.cuh"
#include "gp_launch.h"

namespace gp {

#define GP_PART_DECL(name)                                                              \
  int name(const StageDesc& d, const GridDims& g, const SchemeKey& k,                  \
           cudaStream_t s, cudaEvent_t* ev);
GP_PART_DECL(launch_stage_fp64_p0)
GP_PART_DECL(launch_stage_fp64_p1)
GP_PART_DECL(launch_stage_fp64_p2)
GP_PART_DECL(launch_stage_fp64_p3)
GP_PART_DECL(launch_stage_fp64_p4)
GP_PART_DECL(launch_stage_fp64_p5)
GP_PART_DECL(launch_stage_mixed_p0)
GP_PART_DECL(launch_stage_mixed_p1)
GP_PART_DECL(launch_stage_mixed_p2)
GP_PART_DECL(launch_stage_mixed_p3)
GP_PART_DECL(launch_stage_mixed_p4)
GP_PART_DECL(launch_stage_mixed_p5)

// the unit a scheme is compiled in (GP_PART of gp_launch.cu)
static int part_of(const SchemeKey& k) {
  if (k.physics == PHYS_HD) return 0;
  if (k.physics == PHYS_RMHD) return k.riemann == RS_HLLD ? 2 : 4;
  if (k.physics != PHYS_MHD) return -1;
  if (k.riemann == RS_HLLC || k.riemann == RS_TVDLF) return 3;
  return k.riemann == RS_HLLD && (k.ct == CT_UCT_HLLD || k.ct == CT_UCT_HLL) ? 1 : 5;
}

using LaunchStage = int (*)(const StageDesc&, const GridDims&, const SchemeKey&, cudaStream_t,
                            cudaEvent_t*);

int launch_stage_fp64(const StageDesc& d, const GridDims& g, const SchemeKey& k, cudaStream_t s,
                      cudaEvent_t* ev) {
  static const LaunchStage f[] = {launch_stage_fp64_p0, launch_stage_fp64_p1,
                                  launch_stage_fp64_p2, launch_stage_fp64_p3,
                                  launch_stage_fp64_p4, launch_stage_fp64_p5};
  const int p = part_of(k);
  return p < 0 ? -1 : f[p](d, g, k, s, ev);
}

int launch_stage_mixed(const StageDesc& d, const GridDims& g, const SchemeKey& k, cudaStream_t s,
                       cudaEvent_t* ev) {
  static const LaunchStage f[] = {launch_stage_mixed_p0, launch_stage_mixed_p1,
                                  launch_stage_mixed_p2, launch_stage_mixed_p3,
                                  launch_stage_mixed_p4, launch_stage_mixed_p5};
  const int p = part_of(k);
  return p < 0 ? -1 : f[p](d, g, k, s, ev);
}

}  // namespace gp
