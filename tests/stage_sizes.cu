// Staging areas (bytes a block) of the sweep kernels, for test_stage_sizes.py.
#include "../gpluto_dev_b200/csrc/gp_batch.h"

using namespace gp;

template <int NV, int LIM>
static int row(bool fp32, int which) {
  const int d = fp32 ? (which == 0   ? sweep_m_stage_doubles<NV, LIM, float>()
                        : which == 1 ? sweep_x_stage_doubles<NV, LIM, float, false>()
                                     : sweep_x_stage_doubles<NV, LIM, float, whole_row_form<LIM, float>()>())
                     : (which == 0   ? sweep_m_stage_doubles<NV, LIM, double>()
                                     : sweep_x_stage_doubles<NV, LIM, double, false>());
  return d * (int)sizeof(double);
}

// which: 0 y/z march, 1 x-row in parts, 2 whole x-row
extern "C" int stage_bytes(int nv, int lim, int fp32, int which) {
  if (nv == 8)
    return lim == LIM_PPM ? row<8, LIM_PPM>(fp32, which)
           : lim == LIM_MP5 ? row<8, LIM_MP5>(fp32, which) : row<8, LIM_MC>(fp32, which);
  return lim == LIM_PPM ? row<5, LIM_PPM>(fp32, which)
         : lim == LIM_MP5 ? row<5, LIM_MP5>(fp32, which) : row<5, LIM_MC>(fp32, which);
}

extern "C" int batch_bytes() { return batch_smem_bytes(); }
