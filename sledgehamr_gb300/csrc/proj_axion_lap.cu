/* AxionStringsLap1/2/3 project kernels (projects/AxionStringsLap). */
#define SH_STAGE_CONSTANTS /* the registrations below name StageParams */
#include "../projects/AxionStringsLap/AxionStringsLap.h"
#include "sh_stage.cuh"
SH_DEFINE_PROJECT_OPTIONS(AxionStringsLap1, ::AxionStringsLap1, false, 1, true,
                          &::AxionStringsLap1::StageParams)
SH_DEFINE_PROJECT_OPTIONS(AxionStringsLap2, ::AxionStringsLap2, false, 2, true,
                          &::AxionStringsLap2::StageParams)
SH_DEFINE_PROJECT_OPTIONS(AxionStringsLap3, ::AxionStringsLap3, false, 3, true,
                          &::AxionStringsLap3::StageParams)
