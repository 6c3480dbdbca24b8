/* AxionStrings project kernels (hooks in projects/AxionStrings). */
#define SH_STAGE_CONSTANTS /* the registrations below name StageParams */
#include "../projects/AxionStrings/setup.h"
#include "../projects/AxionStrings/kernels_rhs.h"
#include "../projects/AxionStrings/kernels_tagging.h"
namespace AxionStrings {
SLEDGEHAMR_FINISH_SETUP
}
#include "sh_stage.cuh"
SH_DEFINE_PROJECT_OPTIONS(AxionStrings, ::AxionStrings, true, 2, true,
                          &::AxionStrings::StageParams)
