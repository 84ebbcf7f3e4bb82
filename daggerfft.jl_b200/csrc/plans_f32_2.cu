// Generated by gen_plans.py -- do not edit.
#include "static_plans.h"
namespace dfft {
template __global__ void axis_pass_static<float,1024,3,1,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,3,1,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,9,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,9,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,9,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,9,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,15,1,15>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,15,1,15>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,15,1,15>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,15,1,15>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,24,4,6,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,24,4,6,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,24,4,6,4>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,24,4,6,4>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,32,4,8,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,32,4,8,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,32,4,8,4>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,32,4,8,4>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,42,6,7,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,42,6,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,52,4,13,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,52,4,13,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,64,8,8,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,64,8,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,64,8,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,64,8,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,77,7,11,7>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,77,7,11,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,90,6,15,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,90,6,15,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,16,90,6,15,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,90,6,15,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,104,8,13,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,104,8,13,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,120,10,12,10>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,120,10,12,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,16,120,10,12,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,120,10,12,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,132,11,12,11>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,132,11,12,11>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,150,10,15,10>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,150,10,15,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,16,150,10,15,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,150,10,15,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,168,12,14,12>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,168,12,14,12>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,189,27,7,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,189,27,7,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,208,13,13,16>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,208,13,13,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,231,21,11,7,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,231,21,11,7,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,250,25,10,5,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,250,25,10,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,250,25,10,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,250,25,10,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,273,21,13,7,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,273,21,13,7,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,297,27,11,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,297,27,11,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,324,54,6,6,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,324,54,6,6,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,324,54,6,6,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,324,54,6,6,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,350,35,10,7,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,350,35,10,7,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,375,25,15,5,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,375,25,15,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,375,25,15,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,375,25,15,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,396,36,11,6,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,396,36,11,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,432,36,12,6,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,432,36,12,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,432,36,12,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,432,36,12,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,462,42,11,7,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,462,42,11,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,495,33,15,11,3>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,495,33,15,11,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,525,35,15,7,5>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,525,35,15,7,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,560,56,10,7,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,560,56,10,7,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,594,54,11,6,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,594,54,11,6,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,630,42,15,7,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,630,42,15,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,672,56,12,7,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,672,56,12,7,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,702,54,13,6,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,702,54,13,6,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,729,243,3,3,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,729,243,3,3,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,4,729,243,3,3,3,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,729,243,3,3,3,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,780,60,13,10,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,780,60,13,10,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,825,55,15,11,5>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,825,55,15,11,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,864,72,12,12,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,864,72,12,12,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,8,864,72,12,12,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,864,72,12,12,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,900,60,15,10,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,900,60,15,10,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,8,900,60,15,10,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,900,60,15,10,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,968,88,11,11,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,968,88,11,11,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,1001,77,13,11,7>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,1001,77,13,11,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,1152,96,12,12,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,1152,96,12,12,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,1350,90,15,15,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,1350,90,15,15,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,1620,108,15,12,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,1620,108,15,12,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,2000,200,10,5,5,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,2000,200,10,5,5,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,2304,144,12,12,16>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,2304,144,12,12,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,2700,180,15,15,12>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,2700,180,15,15,12>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,3200,320,10,5,8,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,3200,320,10,5,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,3750,250,15,10,5,5>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,3750,250,15,10,5,5>(const __grid_constant__ PassDesc);
extern const StaticPlan kPlans_f32_2[];
extern const int kPlansCount_f32_2;
const StaticPlan kPlans_f32_2[] = {
  {3, 1, 1, {3}, 1024, (const void*)&axis_pass_static<float,1024,3,1,3>, (const void*)&axis_pass_any<float,1024,false,3,1,3>, nullptr, nullptr, 1024, 0},
  {9, 3, 2, {3,3}, 1024, (const void*)&axis_pass_static<float,1024,9,3,3,3>, (const void*)&axis_pass_any<float,1024,false,9,3,3,3>, (const void*)&axis_pass_pipe<float,1024,false,16,9,3,3,3>, (const void*)&axis_pass_pipe<float,1024,true,0,9,3,3,3>, 1024, 16},
  {15, 1, 1, {15}, 1024, (const void*)&axis_pass_static<float,1024,15,1,15>, (const void*)&axis_pass_any<float,1024,false,15,1,15>, (const void*)&axis_pass_pipe<float,1024,false,16,15,1,15>, (const void*)&axis_pass_pipe<float,1024,true,0,15,1,15>, 1024, 16},
  {24, 4, 2, {6,4}, 1024, (const void*)&axis_pass_static<float,1024,24,4,6,4>, (const void*)&axis_pass_any<float,1024,false,24,4,6,4>, (const void*)&axis_pass_pipe<float,1024,false,16,24,4,6,4>, (const void*)&axis_pass_pipe<float,1024,true,0,24,4,6,4>, 1024, 16},
  {32, 4, 2, {8,4}, 1024, (const void*)&axis_pass_static<float,1024,32,4,8,4>, (const void*)&axis_pass_any<float,1024,false,32,4,8,4>, (const void*)&axis_pass_pipe<float,1024,false,16,32,4,8,4>, (const void*)&axis_pass_pipe<float,1024,true,0,32,4,8,4>, 1024, 16},
  {42, 6, 2, {7,6}, 1024, (const void*)&axis_pass_static<float,1024,42,6,7,6>, (const void*)&axis_pass_any<float,1024,false,42,6,7,6>, nullptr, nullptr, 1024, 0},
  {52, 4, 2, {13,4}, 1024, (const void*)&axis_pass_static<float,1024,52,4,13,4>, (const void*)&axis_pass_any<float,1024,false,52,4,13,4>, nullptr, nullptr, 1024, 0},
  {64, 8, 2, {8,8}, 1024, (const void*)&axis_pass_static<float,1024,64,8,8,8>, (const void*)&axis_pass_any<float,1024,false,64,8,8,8>, (const void*)&axis_pass_pipe<float,1024,false,16,64,8,8,8>, (const void*)&axis_pass_pipe<float,1024,true,0,64,8,8,8>, 1024, 16},
  {77, 7, 2, {11,7}, 1024, (const void*)&axis_pass_static<float,1024,77,7,11,7>, (const void*)&axis_pass_any<float,1024,false,77,7,11,7>, nullptr, nullptr, 1024, 0},
  {90, 6, 2, {15,6}, 512, (const void*)&axis_pass_static<float,512,90,6,15,6>, (const void*)&axis_pass_any<float,512,false,90,6,15,6>, (const void*)&axis_pass_pipe<float,512,false,16,90,6,15,6>, (const void*)&axis_pass_pipe<float,512,true,0,90,6,15,6>, 512, 16},
  {104, 8, 2, {13,8}, 1024, (const void*)&axis_pass_static<float,1024,104,8,13,8>, (const void*)&axis_pass_any<float,1024,false,104,8,13,8>, nullptr, nullptr, 1024, 0},
  {120, 10, 2, {12,10}, 512, (const void*)&axis_pass_static<float,512,120,10,12,10>, (const void*)&axis_pass_any<float,512,false,120,10,12,10>, (const void*)&axis_pass_pipe<float,512,false,16,120,10,12,10>, (const void*)&axis_pass_pipe<float,512,true,0,120,10,12,10>, 512, 16},
  {132, 11, 2, {12,11}, 512, (const void*)&axis_pass_static<float,512,132,11,12,11>, (const void*)&axis_pass_any<float,512,false,132,11,12,11>, nullptr, nullptr, 512, 0},
  {150, 10, 2, {15,10}, 512, (const void*)&axis_pass_static<float,512,150,10,15,10>, (const void*)&axis_pass_any<float,512,false,150,10,15,10>, (const void*)&axis_pass_pipe<float,512,false,16,150,10,15,10>, (const void*)&axis_pass_pipe<float,512,true,0,150,10,15,10>, 512, 16},
  {168, 12, 2, {14,12}, 512, (const void*)&axis_pass_static<float,512,168,12,14,12>, (const void*)&axis_pass_any<float,512,false,168,12,14,12>, nullptr, nullptr, 512, 0},
  {189, 27, 4, {7,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,189,27,7,3,3,3>, (const void*)&axis_pass_any<float,1024,false,189,27,7,3,3,3>, nullptr, nullptr, 1024, 0},
  {208, 13, 2, {13,16}, 512, (const void*)&axis_pass_static<float,512,208,13,13,16>, (const void*)&axis_pass_any<float,512,false,208,13,13,16>, nullptr, nullptr, 512, 0},
  {231, 21, 3, {11,7,3}, 1024, (const void*)&axis_pass_static<float,1024,231,21,11,7,3>, (const void*)&axis_pass_any<float,1024,false,231,21,11,7,3>, nullptr, nullptr, 1024, 0},
  {250, 25, 3, {10,5,5}, 1024, (const void*)&axis_pass_static<float,1024,250,25,10,5,5>, (const void*)&axis_pass_any<float,1024,false,250,25,10,5,5>, (const void*)&axis_pass_pipe<float,1024,false,16,250,25,10,5,5>, (const void*)&axis_pass_pipe<float,1024,true,0,250,25,10,5,5>, 1024, 16},
  {273, 21, 3, {13,7,3}, 1024, (const void*)&axis_pass_static<float,1024,273,21,13,7,3>, (const void*)&axis_pass_any<float,1024,false,273,21,13,7,3>, nullptr, nullptr, 1024, 0},
  {297, 27, 4, {11,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,297,27,11,3,3,3>, (const void*)&axis_pass_any<float,1024,false,297,27,11,3,3,3>, nullptr, nullptr, 1024, 0},
  {324, 54, 4, {6,6,3,3}, 1024, (const void*)&axis_pass_static<float,1024,324,54,6,6,3,3>, (const void*)&axis_pass_any<float,1024,false,324,54,6,6,3,3>, (const void*)&axis_pass_pipe<float,1024,false,16,324,54,6,6,3,3>, (const void*)&axis_pass_pipe<float,1024,true,0,324,54,6,6,3,3>, 1024, 16},
  {350, 35, 3, {10,7,5}, 1024, (const void*)&axis_pass_static<float,1024,350,35,10,7,5>, (const void*)&axis_pass_any<float,1024,false,350,35,10,7,5>, nullptr, nullptr, 1024, 0},
  {375, 25, 3, {15,5,5}, 1024, (const void*)&axis_pass_static<float,1024,375,25,15,5,5>, (const void*)&axis_pass_any<float,1024,false,375,25,15,5,5>, (const void*)&axis_pass_pipe<float,1024,false,16,375,25,15,5,5>, (const void*)&axis_pass_pipe<float,1024,true,0,375,25,15,5,5>, 1024, 16},
  {396, 36, 3, {11,6,6}, 1024, (const void*)&axis_pass_static<float,1024,396,36,11,6,6>, (const void*)&axis_pass_any<float,1024,false,396,36,11,6,6>, nullptr, nullptr, 1024, 0},
  {432, 36, 3, {12,6,6}, 1024, (const void*)&axis_pass_static<float,1024,432,36,12,6,6>, (const void*)&axis_pass_any<float,1024,false,432,36,12,6,6>, (const void*)&axis_pass_pipe<float,1024,false,16,432,36,12,6,6>, (const void*)&axis_pass_pipe<float,1024,true,0,432,36,12,6,6>, 1024, 16},
  {462, 42, 3, {11,7,6}, 1024, (const void*)&axis_pass_static<float,1024,462,42,11,7,6>, (const void*)&axis_pass_any<float,1024,false,462,42,11,7,6>, nullptr, nullptr, 1024, 0},
  {495, 33, 3, {15,11,3}, 512, (const void*)&axis_pass_static<float,512,495,33,15,11,3>, (const void*)&axis_pass_any<float,512,false,495,33,15,11,3>, nullptr, nullptr, 512, 0},
  {525, 35, 3, {15,7,5}, 512, (const void*)&axis_pass_static<float,512,525,35,15,7,5>, (const void*)&axis_pass_any<float,512,false,525,35,15,7,5>, nullptr, nullptr, 512, 0},
  {560, 56, 3, {10,7,8}, 1024, (const void*)&axis_pass_static<float,1024,560,56,10,7,8>, (const void*)&axis_pass_any<float,1024,false,560,56,10,7,8>, nullptr, nullptr, 1024, 0},
  {594, 54, 4, {11,6,3,3}, 1024, (const void*)&axis_pass_static<float,1024,594,54,11,6,3,3>, (const void*)&axis_pass_any<float,1024,false,594,54,11,6,3,3>, nullptr, nullptr, 1024, 0},
  {630, 42, 3, {15,7,6}, 512, (const void*)&axis_pass_static<float,512,630,42,15,7,6>, (const void*)&axis_pass_any<float,512,false,630,42,15,7,6>, nullptr, nullptr, 512, 0},
  {672, 56, 3, {12,7,8}, 1024, (const void*)&axis_pass_static<float,1024,672,56,12,7,8>, (const void*)&axis_pass_any<float,1024,false,672,56,12,7,8>, nullptr, nullptr, 1024, 0},
  {702, 54, 4, {13,6,3,3}, 512, (const void*)&axis_pass_static<float,512,702,54,13,6,3,3>, (const void*)&axis_pass_any<float,512,false,702,54,13,6,3,3>, nullptr, nullptr, 512, 0},
  {729, 243, 6, {3,3,3,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,729,243,3,3,3,3,3,3>, (const void*)&axis_pass_any<float,1024,false,729,243,3,3,3,3,3,3>, (const void*)&axis_pass_pipe<float,1024,false,4,729,243,3,3,3,3,3,3>, (const void*)&axis_pass_pipe<float,1024,true,0,729,243,3,3,3,3,3,3>, 1024, 4},
  {780, 60, 3, {13,10,6}, 512, (const void*)&axis_pass_static<float,512,780,60,13,10,6>, (const void*)&axis_pass_any<float,512,false,780,60,13,10,6>, nullptr, nullptr, 512, 0},
  {825, 55, 3, {15,11,5}, 512, (const void*)&axis_pass_static<float,512,825,55,15,11,5>, (const void*)&axis_pass_any<float,512,false,825,55,15,11,5>, nullptr, nullptr, 512, 0},
  {864, 72, 3, {12,12,6}, 1024, (const void*)&axis_pass_static<float,1024,864,72,12,12,6>, (const void*)&axis_pass_any<float,1024,false,864,72,12,12,6>, (const void*)&axis_pass_pipe<float,1024,false,8,864,72,12,12,6>, (const void*)&axis_pass_pipe<float,1024,true,0,864,72,12,12,6>, 1024, 8},
  {900, 60, 3, {15,10,6}, 512, (const void*)&axis_pass_static<float,512,900,60,15,10,6>, (const void*)&axis_pass_any<float,512,false,900,60,15,10,6>, (const void*)&axis_pass_pipe<float,512,false,8,900,60,15,10,6>, (const void*)&axis_pass_pipe<float,512,true,0,900,60,15,10,6>, 512, 8},
  {968, 88, 3, {11,11,8}, 1024, (const void*)&axis_pass_static<float,1024,968,88,11,11,8>, (const void*)&axis_pass_any<float,1024,false,968,88,11,11,8>, nullptr, nullptr, 1024, 0},
  {1001, 77, 3, {13,11,7}, 512, (const void*)&axis_pass_static<float,512,1001,77,13,11,7>, (const void*)&axis_pass_any<float,512,false,1001,77,13,11,7>, nullptr, nullptr, 512, 0},
  {1152, 96, 3, {12,12,8}, 1024, (const void*)&axis_pass_static<float,1024,1152,96,12,12,8>, (const void*)&axis_pass_any<float,1024,false,1152,96,12,12,8>, nullptr, nullptr, 1024, 0},
  {1350, 90, 3, {15,15,6}, 512, (const void*)&axis_pass_static<float,512,1350,90,15,15,6>, (const void*)&axis_pass_any<float,512,false,1350,90,15,15,6>, nullptr, nullptr, 512, 0},
  {1620, 108, 4, {15,12,3,3}, 512, (const void*)&axis_pass_static<float,512,1620,108,15,12,3,3>, (const void*)&axis_pass_any<float,512,false,1620,108,15,12,3,3>, nullptr, nullptr, 512, 0},
  {2000, 200, 4, {10,5,5,8}, 1024, (const void*)&axis_pass_static<float,1024,2000,200,10,5,5,8>, (const void*)&axis_pass_any<float,1024,false,2000,200,10,5,5,8>, nullptr, nullptr, 1024, 0},
  {2304, 144, 3, {12,12,16}, 512, (const void*)&axis_pass_static<float,512,2304,144,12,12,16>, (const void*)&axis_pass_any<float,512,false,2304,144,12,12,16>, nullptr, nullptr, 512, 0},
  {2700, 180, 3, {15,15,12}, 512, (const void*)&axis_pass_static<float,512,2700,180,15,15,12>, (const void*)&axis_pass_any<float,512,false,2700,180,15,15,12>, nullptr, nullptr, 512, 0},
  {3200, 320, 4, {10,5,8,8}, 1024, (const void*)&axis_pass_static<float,1024,3200,320,10,5,8,8>, (const void*)&axis_pass_any<float,1024,false,3200,320,10,5,8,8>, nullptr, nullptr, 1024, 0},
  {3750, 250, 4, {15,10,5,5}, 512, (const void*)&axis_pass_static<float,512,3750,250,15,10,5,5>, (const void*)&axis_pass_any<float,512,false,3750,250,15,10,5,5>, nullptr, nullptr, 512, 0},
};
const int kPlansCount_f32_2 = 49;
}  // namespace dfft
