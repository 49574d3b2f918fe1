// gt_pcg_fp32.cu -- instances of the persistent Jacobi-PCG: FP32 iteration.
#include "gt_pcg_impl.cuh"

namespace gt {
namespace pcg {

template int cluster_room<float, float, false>(Ctx*, int, ClusterRoom*);
template int run_sliced<float, float, false>(Ctx*, Matrix*, const float*, const double*, double*, double, int, double,
                                    const PRun*, PRun*, int);
template int run_groups_dispatch<float, float, false>(
    Ctx*, Place, int, const std::vector<Matrix*>&, const std::vector<const float*>&,
    const std::vector<const double*>&, const std::vector<double*>&, double, int, double, const std::vector<const PRun*>&,
    std::vector<PRun>&, std::vector<int>&);

}  // namespace pcg
}  // namespace gt
