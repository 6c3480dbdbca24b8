/* MinimalExample and NextToMinimalExample project kernels. */
#define SH_STAGE_CONSTANTS /* the registrations below name StageParams */
#include "../projects/MinimalExample/MinimalExample.h"
#include "../projects/NextToMinimalExample/NextToMinimalExample.h"
#include "sh_stage.cuh"
SH_DEFINE_PROJECT_OPTIONS(MinimalExample, ::MinimalExample, false, 2, true,
                          &::MinimalExample::StageParams)
SH_DEFINE_PROJECT_OPTIONS(NextToMinimalExample, ::NextToMinimalExample, false, 2, true,
                          &::NextToMinimalExample::StageParams)
