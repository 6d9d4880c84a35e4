// The survey solver's kernels for one lane count, MTGPU_SURVEY_SP (set by the
// build: one object per lane count).
#include "survey_impl.cuh"

namespace mtgpu {
namespace sv {

#define MTGPU_OPS_NAME2(n) ops##n
#define MTGPU_OPS_NAME(n) MTGPU_OPS_NAME2(n)
const Ops &MTGPU_OPS_NAME(MTGPU_SURVEY_SP)()
{
    static const Ops o = make_ops<MTGPU_SURVEY_SP>();
    return o;
}

}  // namespace sv
}  // namespace mtgpu
