// Generated by gen_plans.py -- do not edit.
#include "static_plans.h"
namespace dfft {
template __global__ void axis_pass_static<double,1024,3,1,3>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,3,1,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,9,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,9,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,9,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,9,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,15,1,15>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,15,1,15>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,15,1,15>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,15,1,15>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,1024,24,4,6,4>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,24,4,6,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,24,4,6,4>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,24,4,6,4>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,1024,32,4,8,4>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,32,4,8,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,32,4,8,4>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,32,4,8,4>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,42,6,7,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,42,6,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,52,4,13,4>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,52,4,13,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,64,8,8,8>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,64,8,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,64,8,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,64,8,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,77,7,11,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,77,7,11,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,90,6,15,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,90,6,15,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,90,6,15,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,90,6,15,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,104,8,13,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,104,8,13,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,120,10,12,10>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,120,10,12,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,120,10,12,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,120,10,12,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,132,11,12,11>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,132,11,12,11>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,150,10,15,10>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,150,10,15,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,150,10,15,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,150,10,15,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,168,12,14,12>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,168,12,14,12>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,189,27,7,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,189,27,7,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,256,208,13,13,16>(const PassDesc);
template __global__ void axis_pass_any<double,256,false,208,13,13,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,231,21,11,7,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,231,21,11,7,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,250,25,10,5,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,250,25,10,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,250,25,10,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,250,25,10,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,273,21,13,7,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,273,21,13,7,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,297,27,11,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,297,27,11,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,324,54,6,6,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,324,54,6,6,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,324,54,6,6,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,324,54,6,6,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,350,35,10,7,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,350,35,10,7,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,375,25,15,5,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,375,25,15,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,375,25,15,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,375,25,15,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,396,36,11,6,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,396,36,11,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,432,36,12,6,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,432,36,12,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,432,36,12,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,432,36,12,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,462,42,11,7,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,462,42,11,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,495,33,15,11,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,495,33,15,11,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,525,35,15,7,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,525,35,15,7,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,560,56,10,7,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,560,56,10,7,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,594,54,11,6,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,594,54,11,6,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,630,42,15,7,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,630,42,15,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,672,56,12,7,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,672,56,12,7,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,702,54,13,6,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,702,54,13,6,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,729,243,3,3,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,729,243,3,3,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,780,60,13,10,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,780,60,13,10,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,825,55,15,11,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,825,55,15,11,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,864,72,12,12,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,864,72,12,12,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,900,60,15,10,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,900,60,15,10,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,968,88,11,11,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,968,88,11,11,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1001,77,13,11,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1001,77,13,11,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1152,96,12,12,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1152,96,12,12,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1350,90,15,15,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1350,90,15,15,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1620,108,15,12,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1620,108,15,12,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,2000,200,10,5,5,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,2000,200,10,5,5,8>(const __grid_constant__ PassDesc);
extern const StaticPlan kPlans_f64_2[];
extern const int kPlansCount_f64_2;
const StaticPlan kPlans_f64_2[] = {
  {3, 1, 1, {3}, 1024, (const void*)&axis_pass_static<double,1024,3,1,3>, (const void*)&axis_pass_any<double,1024,false,3,1,3>, nullptr, nullptr, 512, 0},
  {9, 3, 2, {3,3}, 1024, (const void*)&axis_pass_static<double,1024,9,3,3,3>, (const void*)&axis_pass_any<double,1024,false,9,3,3,3>, (const void*)&axis_pass_pipe<double,512,false,8,9,3,3,3>, (const void*)&axis_pass_pipe<double,512,true,0,9,3,3,3>, 512, 8},
  {15, 1, 1, {15}, 512, (const void*)&axis_pass_static<double,512,15,1,15>, (const void*)&axis_pass_any<double,512,false,15,1,15>, (const void*)&axis_pass_pipe<double,512,false,8,15,1,15>, (const void*)&axis_pass_pipe<double,512,true,0,15,1,15>, 512, 8},
  {24, 4, 2, {6,4}, 1024, (const void*)&axis_pass_static<double,1024,24,4,6,4>, (const void*)&axis_pass_any<double,1024,false,24,4,6,4>, (const void*)&axis_pass_pipe<double,512,false,8,24,4,6,4>, (const void*)&axis_pass_pipe<double,512,true,0,24,4,6,4>, 512, 8},
  {32, 4, 2, {8,4}, 1024, (const void*)&axis_pass_static<double,1024,32,4,8,4>, (const void*)&axis_pass_any<double,1024,false,32,4,8,4>, (const void*)&axis_pass_pipe<double,512,false,8,32,4,8,4>, (const void*)&axis_pass_pipe<double,512,true,0,32,4,8,4>, 512, 8},
  {42, 6, 2, {7,6}, 512, (const void*)&axis_pass_static<double,512,42,6,7,6>, (const void*)&axis_pass_any<double,512,false,42,6,7,6>, nullptr, nullptr, 512, 0},
  {52, 4, 2, {13,4}, 512, (const void*)&axis_pass_static<double,512,52,4,13,4>, (const void*)&axis_pass_any<double,512,false,52,4,13,4>, nullptr, nullptr, 512, 0},
  {64, 8, 2, {8,8}, 1024, (const void*)&axis_pass_static<double,1024,64,8,8,8>, (const void*)&axis_pass_any<double,1024,false,64,8,8,8>, (const void*)&axis_pass_pipe<double,512,false,8,64,8,8,8>, (const void*)&axis_pass_pipe<double,512,true,0,64,8,8,8>, 512, 8},
  {77, 7, 2, {11,7}, 512, (const void*)&axis_pass_static<double,512,77,7,11,7>, (const void*)&axis_pass_any<double,512,false,77,7,11,7>, nullptr, nullptr, 512, 0},
  {90, 6, 2, {15,6}, 512, (const void*)&axis_pass_static<double,512,90,6,15,6>, (const void*)&axis_pass_any<double,512,false,90,6,15,6>, (const void*)&axis_pass_pipe<double,512,false,8,90,6,15,6>, (const void*)&axis_pass_pipe<double,512,true,0,90,6,15,6>, 512, 8},
  {104, 8, 2, {13,8}, 512, (const void*)&axis_pass_static<double,512,104,8,13,8>, (const void*)&axis_pass_any<double,512,false,104,8,13,8>, nullptr, nullptr, 512, 0},
  {120, 10, 2, {12,10}, 512, (const void*)&axis_pass_static<double,512,120,10,12,10>, (const void*)&axis_pass_any<double,512,false,120,10,12,10>, (const void*)&axis_pass_pipe<double,512,false,8,120,10,12,10>, (const void*)&axis_pass_pipe<double,512,true,0,120,10,12,10>, 512, 8},
  {132, 11, 2, {12,11}, 512, (const void*)&axis_pass_static<double,512,132,11,12,11>, (const void*)&axis_pass_any<double,512,false,132,11,12,11>, nullptr, nullptr, 512, 0},
  {150, 10, 2, {15,10}, 512, (const void*)&axis_pass_static<double,512,150,10,15,10>, (const void*)&axis_pass_any<double,512,false,150,10,15,10>, (const void*)&axis_pass_pipe<double,512,false,8,150,10,15,10>, (const void*)&axis_pass_pipe<double,512,true,0,150,10,15,10>, 512, 8},
  {168, 12, 2, {14,12}, 512, (const void*)&axis_pass_static<double,512,168,12,14,12>, (const void*)&axis_pass_any<double,512,false,168,12,14,12>, nullptr, nullptr, 512, 0},
  {189, 27, 4, {7,3,3,3}, 512, (const void*)&axis_pass_static<double,512,189,27,7,3,3,3>, (const void*)&axis_pass_any<double,512,false,189,27,7,3,3,3>, nullptr, nullptr, 512, 0},
  {208, 13, 2, {13,16}, 256, (const void*)&axis_pass_static<double,256,208,13,13,16>, (const void*)&axis_pass_any<double,256,false,208,13,13,16>, nullptr, nullptr, 256, 0},
  {231, 21, 3, {11,7,3}, 512, (const void*)&axis_pass_static<double,512,231,21,11,7,3>, (const void*)&axis_pass_any<double,512,false,231,21,11,7,3>, nullptr, nullptr, 512, 0},
  {250, 25, 3, {10,5,5}, 512, (const void*)&axis_pass_static<double,512,250,25,10,5,5>, (const void*)&axis_pass_any<double,512,false,250,25,10,5,5>, (const void*)&axis_pass_pipe<double,512,false,8,250,25,10,5,5>, (const void*)&axis_pass_pipe<double,512,true,0,250,25,10,5,5>, 512, 8},
  {273, 21, 3, {13,7,3}, 512, (const void*)&axis_pass_static<double,512,273,21,13,7,3>, (const void*)&axis_pass_any<double,512,false,273,21,13,7,3>, nullptr, nullptr, 512, 0},
  {297, 27, 4, {11,3,3,3}, 512, (const void*)&axis_pass_static<double,512,297,27,11,3,3,3>, (const void*)&axis_pass_any<double,512,false,297,27,11,3,3,3>, nullptr, nullptr, 512, 0},
  {324, 54, 4, {6,6,3,3}, 1024, (const void*)&axis_pass_static<double,1024,324,54,6,6,3,3>, (const void*)&axis_pass_any<double,1024,false,324,54,6,6,3,3>, (const void*)&axis_pass_pipe<double,512,false,8,324,54,6,6,3,3>, (const void*)&axis_pass_pipe<double,512,true,0,324,54,6,6,3,3>, 512, 8},
  {350, 35, 3, {10,7,5}, 512, (const void*)&axis_pass_static<double,512,350,35,10,7,5>, (const void*)&axis_pass_any<double,512,false,350,35,10,7,5>, nullptr, nullptr, 512, 0},
  {375, 25, 3, {15,5,5}, 512, (const void*)&axis_pass_static<double,512,375,25,15,5,5>, (const void*)&axis_pass_any<double,512,false,375,25,15,5,5>, (const void*)&axis_pass_pipe<double,512,false,8,375,25,15,5,5>, (const void*)&axis_pass_pipe<double,512,true,0,375,25,15,5,5>, 512, 8},
  {396, 36, 3, {11,6,6}, 512, (const void*)&axis_pass_static<double,512,396,36,11,6,6>, (const void*)&axis_pass_any<double,512,false,396,36,11,6,6>, nullptr, nullptr, 512, 0},
  {432, 36, 3, {12,6,6}, 512, (const void*)&axis_pass_static<double,512,432,36,12,6,6>, (const void*)&axis_pass_any<double,512,false,432,36,12,6,6>, (const void*)&axis_pass_pipe<double,512,false,8,432,36,12,6,6>, (const void*)&axis_pass_pipe<double,512,true,0,432,36,12,6,6>, 512, 8},
  {462, 42, 3, {11,7,6}, 512, (const void*)&axis_pass_static<double,512,462,42,11,7,6>, (const void*)&axis_pass_any<double,512,false,462,42,11,7,6>, nullptr, nullptr, 512, 0},
  {495, 33, 3, {15,11,3}, 512, (const void*)&axis_pass_static<double,512,495,33,15,11,3>, (const void*)&axis_pass_any<double,512,false,495,33,15,11,3>, nullptr, nullptr, 512, 0},
  {525, 35, 3, {15,7,5}, 512, (const void*)&axis_pass_static<double,512,525,35,15,7,5>, (const void*)&axis_pass_any<double,512,false,525,35,15,7,5>, nullptr, nullptr, 512, 0},
  {560, 56, 3, {10,7,8}, 512, (const void*)&axis_pass_static<double,512,560,56,10,7,8>, (const void*)&axis_pass_any<double,512,false,560,56,10,7,8>, nullptr, nullptr, 512, 0},
  {594, 54, 4, {11,6,3,3}, 512, (const void*)&axis_pass_static<double,512,594,54,11,6,3,3>, (const void*)&axis_pass_any<double,512,false,594,54,11,6,3,3>, nullptr, nullptr, 512, 0},
  {630, 42, 3, {15,7,6}, 512, (const void*)&axis_pass_static<double,512,630,42,15,7,6>, (const void*)&axis_pass_any<double,512,false,630,42,15,7,6>, nullptr, nullptr, 512, 0},
  {672, 56, 3, {12,7,8}, 512, (const void*)&axis_pass_static<double,512,672,56,12,7,8>, (const void*)&axis_pass_any<double,512,false,672,56,12,7,8>, nullptr, nullptr, 512, 0},
  {702, 54, 4, {13,6,3,3}, 512, (const void*)&axis_pass_static<double,512,702,54,13,6,3,3>, (const void*)&axis_pass_any<double,512,false,702,54,13,6,3,3>, nullptr, nullptr, 512, 0},
  {729, 243, 6, {3,3,3,3,3,3}, 1024, (const void*)&axis_pass_static<double,1024,729,243,3,3,3,3,3,3>, (const void*)&axis_pass_any<double,1024,false,729,243,3,3,3,3,3,3>, nullptr, nullptr, 512, 0},
  {780, 60, 3, {13,10,6}, 512, (const void*)&axis_pass_static<double,512,780,60,13,10,6>, (const void*)&axis_pass_any<double,512,false,780,60,13,10,6>, nullptr, nullptr, 512, 0},
  {825, 55, 3, {15,11,5}, 512, (const void*)&axis_pass_static<double,512,825,55,15,11,5>, (const void*)&axis_pass_any<double,512,false,825,55,15,11,5>, nullptr, nullptr, 512, 0},
  {864, 72, 3, {12,12,6}, 512, (const void*)&axis_pass_static<double,512,864,72,12,12,6>, (const void*)&axis_pass_any<double,512,false,864,72,12,12,6>, nullptr, nullptr, 512, 0},
  {900, 60, 3, {15,10,6}, 512, (const void*)&axis_pass_static<double,512,900,60,15,10,6>, (const void*)&axis_pass_any<double,512,false,900,60,15,10,6>, nullptr, nullptr, 512, 0},
  {968, 88, 3, {11,11,8}, 512, (const void*)&axis_pass_static<double,512,968,88,11,11,8>, (const void*)&axis_pass_any<double,512,false,968,88,11,11,8>, nullptr, nullptr, 512, 0},
  {1001, 77, 3, {13,11,7}, 512, (const void*)&axis_pass_static<double,512,1001,77,13,11,7>, (const void*)&axis_pass_any<double,512,false,1001,77,13,11,7>, nullptr, nullptr, 512, 0},
  {1152, 96, 3, {12,12,8}, 512, (const void*)&axis_pass_static<double,512,1152,96,12,12,8>, (const void*)&axis_pass_any<double,512,false,1152,96,12,12,8>, nullptr, nullptr, 512, 0},
  {1350, 90, 3, {15,15,6}, 512, (const void*)&axis_pass_static<double,512,1350,90,15,15,6>, (const void*)&axis_pass_any<double,512,false,1350,90,15,15,6>, nullptr, nullptr, 512, 0},
  {1620, 108, 4, {15,12,3,3}, 512, (const void*)&axis_pass_static<double,512,1620,108,15,12,3,3>, (const void*)&axis_pass_any<double,512,false,1620,108,15,12,3,3>, nullptr, nullptr, 512, 0},
  {2000, 200, 4, {10,5,5,8}, 512, (const void*)&axis_pass_static<double,512,2000,200,10,5,5,8>, (const void*)&axis_pass_any<double,512,false,2000,200,10,5,5,8>, nullptr, nullptr, 512, 0},
};
const int kPlansCount_f64_2 = 45;
}  // namespace dfft
