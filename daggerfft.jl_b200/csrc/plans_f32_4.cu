// Generated by gen_plans.py -- do not edit.
#include "static_plans.h"
namespace dfft {
template __global__ void axis_pass_static<float,1024,5,1,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,5,1,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,11,1,11>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,11,1,11>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,18,3,6,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,18,3,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,18,3,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,18,3,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,26,2,13,2>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,26,2,13,2>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,35,5,7,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,35,5,7,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,45,3,15,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,45,3,15,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,45,3,15,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,45,3,15,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,55,5,11,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,55,5,11,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,66,6,11,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,66,6,11,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,80,8,10,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,80,8,10,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,80,8,10,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,80,8,10,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,96,8,12,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,96,8,12,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,96,8,12,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,96,8,12,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,108,18,6,6,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,108,18,6,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,108,18,6,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,108,18,6,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,125,25,5,5,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,125,25,5,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,125,25,5,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,125,25,5,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,140,10,14,10>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,140,10,14,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,156,12,13,12>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,156,12,13,12>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,175,25,7,5,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,175,25,7,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,195,13,15,13>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,195,13,15,13>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,216,36,6,6,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,216,36,6,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,216,36,6,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,216,36,6,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,240,15,15,16>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,240,15,15,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,16,240,15,15,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,240,15,15,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,256,16,16,16>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,256,16,16,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,256,16,16,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,256,16,16,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,280,35,7,5,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,280,35,7,5,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,308,28,11,7,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,308,28,11,7,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,330,30,11,6,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,330,30,11,6,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,352,32,11,8,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,352,32,11,8,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,384,48,6,8,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,384,48,6,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,384,48,6,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,384,48,6,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,405,27,15,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,405,27,15,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,405,27,15,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,405,27,15,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,441,63,7,7,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,441,63,7,7,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,480,48,10,6,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,480,48,10,6,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,480,48,10,6,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,480,48,10,6,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,504,42,12,7,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,504,42,12,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,539,49,11,7,7>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,539,49,11,7,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,572,44,13,11,4>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,572,44,13,11,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,605,55,11,11,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,605,55,11,11,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,640,64,10,8,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,640,64,10,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,8,640,64,10,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,640,64,10,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,676,52,13,13,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,676,52,13,13,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,715,55,13,11,5>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,715,55,13,11,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,750,50,15,10,5>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,750,50,15,10,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,8,750,50,15,10,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,750,50,15,10,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,792,66,12,11,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,792,66,12,11,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,840,70,12,10,7>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,840,70,12,10,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,880,80,11,10,8>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,880,80,11,10,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,924,77,12,11,7>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,924,77,12,11,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,975,65,15,13,5>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,975,65,15,13,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,1014,78,13,13,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,1014,78,13,13,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,1215,81,15,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,1215,81,15,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,1458,243,6,3,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,1458,243,6,3,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,1800,120,15,12,10>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,1800,120,15,12,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,2048,128,16,16,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,2048,128,16,16,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,2430,162,15,6,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,2430,162,15,6,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,2916,486,6,6,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,2916,486,6,6,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,3375,225,15,15,15>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,3375,225,15,15,15>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,3888,648,6,6,6,6,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,3888,648,6,6,6,6,3>(const __grid_constant__ PassDesc);
extern const StaticPlan kPlans_f32_4[];
extern const int kPlansCount_f32_4;
const StaticPlan kPlans_f32_4[] = {
  {5, 1, 1, {5}, 1024, (const void*)&axis_pass_static<float,1024,5,1,5>, (const void*)&axis_pass_any<float,1024,false,5,1,5>, nullptr, nullptr, 1024, 0},
  {11, 1, 1, {11}, 1024, (const void*)&axis_pass_static<float,1024,11,1,11>, (const void*)&axis_pass_any<float,1024,false,11,1,11>, nullptr, nullptr, 1024, 0},
  {18, 3, 2, {6,3}, 1024, (const void*)&axis_pass_static<float,1024,18,3,6,3>, (const void*)&axis_pass_any<float,1024,false,18,3,6,3>, (const void*)&axis_pass_pipe<float,1024,false,16,18,3,6,3>, (const void*)&axis_pass_pipe<float,1024,true,0,18,3,6,3>, 1024, 16},
  {26, 2, 2, {13,2}, 1024, (const void*)&axis_pass_static<float,1024,26,2,13,2>, (const void*)&axis_pass_any<float,1024,false,26,2,13,2>, nullptr, nullptr, 1024, 0},
  {35, 5, 2, {7,5}, 1024, (const void*)&axis_pass_static<float,1024,35,5,7,5>, (const void*)&axis_pass_any<float,1024,false,35,5,7,5>, nullptr, nullptr, 1024, 0},
  {45, 3, 2, {15,3}, 1024, (const void*)&axis_pass_static<float,1024,45,3,15,3>, (const void*)&axis_pass_any<float,1024,false,45,3,15,3>, (const void*)&axis_pass_pipe<float,1024,false,16,45,3,15,3>, (const void*)&axis_pass_pipe<float,1024,true,0,45,3,15,3>, 1024, 16},
  {55, 5, 2, {11,5}, 1024, (const void*)&axis_pass_static<float,1024,55,5,11,5>, (const void*)&axis_pass_any<float,1024,false,55,5,11,5>, nullptr, nullptr, 1024, 0},
  {66, 6, 2, {11,6}, 1024, (const void*)&axis_pass_static<float,1024,66,6,11,6>, (const void*)&axis_pass_any<float,1024,false,66,6,11,6>, nullptr, nullptr, 1024, 0},
  {80, 8, 2, {10,8}, 1024, (const void*)&axis_pass_static<float,1024,80,8,10,8>, (const void*)&axis_pass_any<float,1024,false,80,8,10,8>, (const void*)&axis_pass_pipe<float,1024,false,16,80,8,10,8>, (const void*)&axis_pass_pipe<float,1024,true,0,80,8,10,8>, 1024, 16},
  {96, 8, 2, {12,8}, 1024, (const void*)&axis_pass_static<float,1024,96,8,12,8>, (const void*)&axis_pass_any<float,1024,false,96,8,12,8>, (const void*)&axis_pass_pipe<float,1024,false,16,96,8,12,8>, (const void*)&axis_pass_pipe<float,1024,true,0,96,8,12,8>, 1024, 16},
  {108, 18, 3, {6,6,3}, 1024, (const void*)&axis_pass_static<float,1024,108,18,6,6,3>, (const void*)&axis_pass_any<float,1024,false,108,18,6,6,3>, (const void*)&axis_pass_pipe<float,1024,false,16,108,18,6,6,3>, (const void*)&axis_pass_pipe<float,1024,true,0,108,18,6,6,3>, 1024, 16},
  {125, 25, 3, {5,5,5}, 1024, (const void*)&axis_pass_static<float,1024,125,25,5,5,5>, (const void*)&axis_pass_any<float,1024,false,125,25,5,5,5>, (const void*)&axis_pass_pipe<float,1024,false,16,125,25,5,5,5>, (const void*)&axis_pass_pipe<float,1024,true,0,125,25,5,5,5>, 1024, 16},
  {140, 10, 2, {14,10}, 512, (const void*)&axis_pass_static<float,512,140,10,14,10>, (const void*)&axis_pass_any<float,512,false,140,10,14,10>, nullptr, nullptr, 512, 0},
  {156, 12, 2, {13,12}, 512, (const void*)&axis_pass_static<float,512,156,12,13,12>, (const void*)&axis_pass_any<float,512,false,156,12,13,12>, nullptr, nullptr, 512, 0},
  {175, 25, 3, {7,5,5}, 1024, (const void*)&axis_pass_static<float,1024,175,25,7,5,5>, (const void*)&axis_pass_any<float,1024,false,175,25,7,5,5>, nullptr, nullptr, 1024, 0},
  {195, 13, 2, {15,13}, 512, (const void*)&axis_pass_static<float,512,195,13,15,13>, (const void*)&axis_pass_any<float,512,false,195,13,15,13>, nullptr, nullptr, 512, 0},
  {216, 36, 3, {6,6,6}, 1024, (const void*)&axis_pass_static<float,1024,216,36,6,6,6>, (const void*)&axis_pass_any<float,1024,false,216,36,6,6,6>, (const void*)&axis_pass_pipe<float,1024,false,16,216,36,6,6,6>, (const void*)&axis_pass_pipe<float,1024,true,0,216,36,6,6,6>, 1024, 16},
  {240, 15, 2, {15,16}, 512, (const void*)&axis_pass_static<float,512,240,15,15,16>, (const void*)&axis_pass_any<float,512,false,240,15,15,16>, (const void*)&axis_pass_pipe<float,512,false,16,240,15,15,16>, (const void*)&axis_pass_pipe<float,512,true,0,240,15,15,16>, 512, 16},
  {256, 16, 2, {16,16}, 1024, (const void*)&axis_pass_static<float,1024,256,16,16,16>, (const void*)&axis_pass_any<float,1024,false,256,16,16,16>, (const void*)&axis_pass_pipe<float,1024,false,16,256,16,16,16>, (const void*)&axis_pass_pipe<float,1024,true,0,256,16,16,16>, 1024, 16},
  {280, 35, 3, {7,5,8}, 1024, (const void*)&axis_pass_static<float,1024,280,35,7,5,8>, (const void*)&axis_pass_any<float,1024,false,280,35,7,5,8>, nullptr, nullptr, 1024, 0},
  {308, 28, 3, {11,7,4}, 1024, (const void*)&axis_pass_static<float,1024,308,28,11,7,4>, (const void*)&axis_pass_any<float,1024,false,308,28,11,7,4>, nullptr, nullptr, 1024, 0},
  {330, 30, 3, {11,6,5}, 1024, (const void*)&axis_pass_static<float,1024,330,30,11,6,5>, (const void*)&axis_pass_any<float,1024,false,330,30,11,6,5>, nullptr, nullptr, 1024, 0},
  {352, 32, 3, {11,8,4}, 1024, (const void*)&axis_pass_static<float,1024,352,32,11,8,4>, (const void*)&axis_pass_any<float,1024,false,352,32,11,8,4>, nullptr, nullptr, 1024, 0},
  {384, 48, 3, {6,8,8}, 1024, (const void*)&axis_pass_static<float,1024,384,48,6,8,8>, (const void*)&axis_pass_any<float,1024,false,384,48,6,8,8>, (const void*)&axis_pass_pipe<float,1024,false,16,384,48,6,8,8>, (const void*)&axis_pass_pipe<float,1024,true,0,384,48,6,8,8>, 1024, 16},
  {405, 27, 4, {15,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,405,27,15,3,3,3>, (const void*)&axis_pass_any<float,1024,false,405,27,15,3,3,3>, (const void*)&axis_pass_pipe<float,1024,false,16,405,27,15,3,3,3>, (const void*)&axis_pass_pipe<float,1024,true,0,405,27,15,3,3,3>, 1024, 16},
  {441, 63, 4, {7,7,3,3}, 1024, (const void*)&axis_pass_static<float,1024,441,63,7,7,3,3>, (const void*)&axis_pass_any<float,1024,false,441,63,7,7,3,3>, nullptr, nullptr, 1024, 0},
  {480, 48, 3, {10,6,8}, 1024, (const void*)&axis_pass_static<float,1024,480,48,10,6,8>, (const void*)&axis_pass_any<float,1024,false,480,48,10,6,8>, (const void*)&axis_pass_pipe<float,1024,false,16,480,48,10,6,8>, (const void*)&axis_pass_pipe<float,1024,true,0,480,48,10,6,8>, 1024, 16},
  {504, 42, 3, {12,7,6}, 1024, (const void*)&axis_pass_static<float,1024,504,42,12,7,6>, (const void*)&axis_pass_any<float,1024,false,504,42,12,7,6>, nullptr, nullptr, 1024, 0},
  {539, 49, 3, {11,7,7}, 1024, (const void*)&axis_pass_static<float,1024,539,49,11,7,7>, (const void*)&axis_pass_any<float,1024,false,539,49,11,7,7>, nullptr, nullptr, 1024, 0},
  {572, 44, 3, {13,11,4}, 512, (const void*)&axis_pass_static<float,512,572,44,13,11,4>, (const void*)&axis_pass_any<float,512,false,572,44,13,11,4>, nullptr, nullptr, 512, 0},
  {605, 55, 3, {11,11,5}, 1024, (const void*)&axis_pass_static<float,1024,605,55,11,11,5>, (const void*)&axis_pass_any<float,1024,false,605,55,11,11,5>, nullptr, nullptr, 1024, 0},
  {640, 64, 3, {10,8,8}, 1024, (const void*)&axis_pass_static<float,1024,640,64,10,8,8>, (const void*)&axis_pass_any<float,1024,false,640,64,10,8,8>, (const void*)&axis_pass_pipe<float,1024,false,8,640,64,10,8,8>, (const void*)&axis_pass_pipe<float,1024,true,0,640,64,10,8,8>, 1024, 8},
  {676, 52, 3, {13,13,4}, 1024, (const void*)&axis_pass_static<float,1024,676,52,13,13,4>, (const void*)&axis_pass_any<float,1024,false,676,52,13,13,4>, nullptr, nullptr, 1024, 0},
  {715, 55, 3, {13,11,5}, 512, (const void*)&axis_pass_static<float,512,715,55,13,11,5>, (const void*)&axis_pass_any<float,512,false,715,55,13,11,5>, nullptr, nullptr, 512, 0},
  {750, 50, 3, {15,10,5}, 512, (const void*)&axis_pass_static<float,512,750,50,15,10,5>, (const void*)&axis_pass_any<float,512,false,750,50,15,10,5>, (const void*)&axis_pass_pipe<float,512,false,8,750,50,15,10,5>, (const void*)&axis_pass_pipe<float,512,true,0,750,50,15,10,5>, 512, 8},
  {792, 66, 3, {12,11,6}, 512, (const void*)&axis_pass_static<float,512,792,66,12,11,6>, (const void*)&axis_pass_any<float,512,false,792,66,12,11,6>, nullptr, nullptr, 512, 0},
  {840, 70, 3, {12,10,7}, 512, (const void*)&axis_pass_static<float,512,840,70,12,10,7>, (const void*)&axis_pass_any<float,512,false,840,70,12,10,7>, nullptr, nullptr, 512, 0},
  {880, 80, 3, {11,10,8}, 512, (const void*)&axis_pass_static<float,512,880,80,11,10,8>, (const void*)&axis_pass_any<float,512,false,880,80,11,10,8>, nullptr, nullptr, 512, 0},
  {924, 77, 3, {12,11,7}, 512, (const void*)&axis_pass_static<float,512,924,77,12,11,7>, (const void*)&axis_pass_any<float,512,false,924,77,12,11,7>, nullptr, nullptr, 512, 0},
  {975, 65, 3, {15,13,5}, 512, (const void*)&axis_pass_static<float,512,975,65,15,13,5>, (const void*)&axis_pass_any<float,512,false,975,65,15,13,5>, nullptr, nullptr, 512, 0},
  {1014, 78, 3, {13,13,6}, 512, (const void*)&axis_pass_static<float,512,1014,78,13,13,6>, (const void*)&axis_pass_any<float,512,false,1014,78,13,13,6>, nullptr, nullptr, 512, 0},
  {1215, 81, 5, {15,3,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,1215,81,15,3,3,3,3>, (const void*)&axis_pass_any<float,1024,false,1215,81,15,3,3,3,3>, nullptr, nullptr, 1024, 0},
  {1458, 243, 6, {6,3,3,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,1458,243,6,3,3,3,3,3>, (const void*)&axis_pass_any<float,1024,false,1458,243,6,3,3,3,3,3>, nullptr, nullptr, 1024, 0},
  {1800, 120, 3, {15,12,10}, 512, (const void*)&axis_pass_static<float,512,1800,120,15,12,10>, (const void*)&axis_pass_any<float,512,false,1800,120,15,12,10>, nullptr, nullptr, 512, 0},
  {2048, 128, 3, {16,16,8}, 1024, (const void*)&axis_pass_static<float,1024,2048,128,16,16,8>, (const void*)&axis_pass_any<float,1024,false,2048,128,16,16,8>, nullptr, nullptr, 1024, 0},
  {2430, 162, 5, {15,6,3,3,3}, 512, (const void*)&axis_pass_static<float,512,2430,162,15,6,3,3,3>, (const void*)&axis_pass_any<float,512,false,2430,162,15,6,3,3,3>, nullptr, nullptr, 512, 0},
  {2916, 486, 6, {6,6,3,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,2916,486,6,6,3,3,3,3>, (const void*)&axis_pass_any<float,1024,false,2916,486,6,6,3,3,3,3>, nullptr, nullptr, 1024, 0},
  {3375, 225, 3, {15,15,15}, 1024, (const void*)&axis_pass_static<float,1024,3375,225,15,15,15>, (const void*)&axis_pass_any<float,1024,false,3375,225,15,15,15>, nullptr, nullptr, 1024, 0},
  {3888, 648, 5, {6,6,6,6,3}, 1024, (const void*)&axis_pass_static<float,1024,3888,648,6,6,6,6,3>, (const void*)&axis_pass_any<float,1024,false,3888,648,6,6,6,6,3>, nullptr, nullptr, 1024, 0},
};
const int kPlansCount_f32_4 = 49;
}  // namespace dfft
