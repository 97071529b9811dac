// fsl_dyn32.cu -- the dynamic Smagorinsky procedure in FP32 for the FP32-bulk
// path (filters, Leonard stress, strain rates and coefficient in FP32 from
// the FP64 state; mu_SGS written as the FP32 field the stage kernel reads).
#include <algorithm>

#define FSL_CHK_UNIT FSL_CHK_DYN32
#include "fsl_dyn.cuh"

FSL_CHK_EXPORT(dyn32)

namespace fsl {

long long dyn_units(const Grid &g) { return dyn::march_units(g); }
int dyn_cut(const Grid &g, int sms) { return dyn::march_cut(g, sms); }

int launch_dynsmag32(Ctx &c, const double *U, float *cd)
{
    prof_begin(c, FSL_K_SGS);
    const int e = dyn::march<float>(c.g, c.k, U, c.mu32, cd, c.dyn_cut, c.dyn_seg, c.stream);
    prof_end(c, FSL_K_SGS, 1);
    if (!e) return FSL_OK;
    c.err = "dynamic procedure: kernel launch";
    return FSL_ERR_CUDA;
}

} // namespace fsl
