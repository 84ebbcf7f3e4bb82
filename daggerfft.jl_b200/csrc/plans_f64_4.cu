// Generated by gen_plans.py -- do not edit.
#include "static_plans.h"
namespace dfft {
template __global__ void axis_pass_static<double,1024,5,1,5>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,5,1,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,11,1,11>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,11,1,11>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,18,3,6,3>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,18,3,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,18,3,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,18,3,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,26,2,13,2>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,26,2,13,2>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,35,5,7,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,35,5,7,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,45,3,15,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,45,3,15,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,45,3,15,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,45,3,15,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,55,5,11,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,55,5,11,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,66,6,11,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,66,6,11,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,80,8,10,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,80,8,10,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,80,8,10,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,80,8,10,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,96,8,12,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,96,8,12,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,96,8,12,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,96,8,12,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,1024,108,18,6,6,3>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,108,18,6,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,108,18,6,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,108,18,6,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,1024,125,25,5,5,5>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,125,25,5,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,125,25,5,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,125,25,5,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,140,10,14,10>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,140,10,14,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,156,12,13,12>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,156,12,13,12>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,175,25,7,5,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,175,25,7,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,256,195,13,15,13>(const PassDesc);
template __global__ void axis_pass_any<double,256,false,195,13,15,13>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,216,36,6,6,6>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,216,36,6,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,216,36,6,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,216,36,6,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,256,240,15,15,16>(const PassDesc);
template __global__ void axis_pass_any<double,256,false,240,15,15,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,256,false,8,240,15,15,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,256,true,0,240,15,15,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,256,16,16,16>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,256,16,16,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,256,16,16,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,256,16,16,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,280,35,7,5,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,280,35,7,5,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,308,28,11,7,4>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,308,28,11,7,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,330,30,11,6,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,330,30,11,6,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,352,32,11,8,4>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,352,32,11,8,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,384,48,6,8,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,384,48,6,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,384,48,6,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,384,48,6,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,405,27,15,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,405,27,15,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,405,27,15,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,405,27,15,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,441,63,7,7,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,441,63,7,7,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,480,48,10,6,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,480,48,10,6,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,480,48,10,6,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,480,48,10,6,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,504,42,12,7,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,504,42,12,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,539,49,11,7,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,539,49,11,7,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,572,44,13,11,4>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,572,44,13,11,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,605,55,11,11,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,605,55,11,11,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,640,64,10,8,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,640,64,10,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,676,52,13,13,4>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,676,52,13,13,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,715,55,13,11,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,715,55,13,11,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,750,50,15,10,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,750,50,15,10,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,792,66,12,11,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,792,66,12,11,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,840,70,12,10,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,840,70,12,10,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,880,80,11,10,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,880,80,11,10,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,924,77,12,11,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,924,77,12,11,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,256,975,65,15,13,5>(const PassDesc);
template __global__ void axis_pass_any<double,256,false,975,65,15,13,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1014,78,13,13,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1014,78,13,13,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1215,81,15,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1215,81,15,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,1458,243,6,3,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,1458,243,6,3,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1800,120,15,12,10>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1800,120,15,12,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,2048,128,16,16,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,2048,128,16,16,8>(const __grid_constant__ PassDesc);
extern const StaticPlan kPlans_f64_4[];
extern const int kPlansCount_f64_4;
const StaticPlan kPlans_f64_4[] = {
  {5, 1, 1, {5}, 1024, (const void*)&axis_pass_static<double,1024,5,1,5>, (const void*)&axis_pass_any<double,1024,false,5,1,5>, nullptr, nullptr, 512, 0},
  {11, 1, 1, {11}, 512, (const void*)&axis_pass_static<double,512,11,1,11>, (const void*)&axis_pass_any<double,512,false,11,1,11>, nullptr, nullptr, 512, 0},
  {18, 3, 2, {6,3}, 1024, (const void*)&axis_pass_static<double,1024,18,3,6,3>, (const void*)&axis_pass_any<double,1024,false,18,3,6,3>, (const void*)&axis_pass_pipe<double,512,false,8,18,3,6,3>, (const void*)&axis_pass_pipe<double,512,true,0,18,3,6,3>, 512, 8},
  {26, 2, 2, {13,2}, 512, (const void*)&axis_pass_static<double,512,26,2,13,2>, (const void*)&axis_pass_any<double,512,false,26,2,13,2>, nullptr, nullptr, 512, 0},
  {35, 5, 2, {7,5}, 512, (const void*)&axis_pass_static<double,512,35,5,7,5>, (const void*)&axis_pass_any<double,512,false,35,5,7,5>, nullptr, nullptr, 512, 0},
  {45, 3, 2, {15,3}, 512, (const void*)&axis_pass_static<double,512,45,3,15,3>, (const void*)&axis_pass_any<double,512,false,45,3,15,3>, (const void*)&axis_pass_pipe<double,512,false,8,45,3,15,3>, (const void*)&axis_pass_pipe<double,512,true,0,45,3,15,3>, 512, 8},
  {55, 5, 2, {11,5}, 512, (const void*)&axis_pass_static<double,512,55,5,11,5>, (const void*)&axis_pass_any<double,512,false,55,5,11,5>, nullptr, nullptr, 512, 0},
  {66, 6, 2, {11,6}, 512, (const void*)&axis_pass_static<double,512,66,6,11,6>, (const void*)&axis_pass_any<double,512,false,66,6,11,6>, nullptr, nullptr, 512, 0},
  {80, 8, 2, {10,8}, 512, (const void*)&axis_pass_static<double,512,80,8,10,8>, (const void*)&axis_pass_any<double,512,false,80,8,10,8>, (const void*)&axis_pass_pipe<double,512,false,8,80,8,10,8>, (const void*)&axis_pass_pipe<double,512,true,0,80,8,10,8>, 512, 8},
  {96, 8, 2, {12,8}, 512, (const void*)&axis_pass_static<double,512,96,8,12,8>, (const void*)&axis_pass_any<double,512,false,96,8,12,8>, (const void*)&axis_pass_pipe<double,512,false,8,96,8,12,8>, (const void*)&axis_pass_pipe<double,512,true,0,96,8,12,8>, 512, 8},
  {108, 18, 3, {6,6,3}, 1024, (const void*)&axis_pass_static<double,1024,108,18,6,6,3>, (const void*)&axis_pass_any<double,1024,false,108,18,6,6,3>, (const void*)&axis_pass_pipe<double,512,false,8,108,18,6,6,3>, (const void*)&axis_pass_pipe<double,512,true,0,108,18,6,6,3>, 512, 8},
  {125, 25, 3, {5,5,5}, 1024, (const void*)&axis_pass_static<double,1024,125,25,5,5,5>, (const void*)&axis_pass_any<double,1024,false,125,25,5,5,5>, (const void*)&axis_pass_pipe<double,512,false,8,125,25,5,5,5>, (const void*)&axis_pass_pipe<double,512,true,0,125,25,5,5,5>, 512, 8},
  {140, 10, 2, {14,10}, 512, (const void*)&axis_pass_static<double,512,140,10,14,10>, (const void*)&axis_pass_any<double,512,false,140,10,14,10>, nullptr, nullptr, 512, 0},
  {156, 12, 2, {13,12}, 512, (const void*)&axis_pass_static<double,512,156,12,13,12>, (const void*)&axis_pass_any<double,512,false,156,12,13,12>, nullptr, nullptr, 512, 0},
  {175, 25, 3, {7,5,5}, 512, (const void*)&axis_pass_static<double,512,175,25,7,5,5>, (const void*)&axis_pass_any<double,512,false,175,25,7,5,5>, nullptr, nullptr, 512, 0},
  {195, 13, 2, {15,13}, 256, (const void*)&axis_pass_static<double,256,195,13,15,13>, (const void*)&axis_pass_any<double,256,false,195,13,15,13>, nullptr, nullptr, 256, 0},
  {216, 36, 3, {6,6,6}, 1024, (const void*)&axis_pass_static<double,1024,216,36,6,6,6>, (const void*)&axis_pass_any<double,1024,false,216,36,6,6,6>, (const void*)&axis_pass_pipe<double,512,false,8,216,36,6,6,6>, (const void*)&axis_pass_pipe<double,512,true,0,216,36,6,6,6>, 512, 8},
  {240, 15, 2, {15,16}, 256, (const void*)&axis_pass_static<double,256,240,15,15,16>, (const void*)&axis_pass_any<double,256,false,240,15,15,16>, (const void*)&axis_pass_pipe<double,256,false,8,240,15,15,16>, (const void*)&axis_pass_pipe<double,256,true,0,240,15,15,16>, 256, 8},
  {256, 16, 2, {16,16}, 512, (const void*)&axis_pass_static<double,512,256,16,16,16>, (const void*)&axis_pass_any<double,512,false,256,16,16,16>, (const void*)&axis_pass_pipe<double,512,false,8,256,16,16,16>, (const void*)&axis_pass_pipe<double,512,true,0,256,16,16,16>, 512, 8},
  {280, 35, 3, {7,5,8}, 512, (const void*)&axis_pass_static<double,512,280,35,7,5,8>, (const void*)&axis_pass_any<double,512,false,280,35,7,5,8>, nullptr, nullptr, 512, 0},
  {308, 28, 3, {11,7,4}, 512, (const void*)&axis_pass_static<double,512,308,28,11,7,4>, (const void*)&axis_pass_any<double,512,false,308,28,11,7,4>, nullptr, nullptr, 512, 0},
  {330, 30, 3, {11,6,5}, 512, (const void*)&axis_pass_static<double,512,330,30,11,6,5>, (const void*)&axis_pass_any<double,512,false,330,30,11,6,5>, nullptr, nullptr, 512, 0},
  {352, 32, 3, {11,8,4}, 512, (const void*)&axis_pass_static<double,512,352,32,11,8,4>, (const void*)&axis_pass_any<double,512,false,352,32,11,8,4>, nullptr, nullptr, 512, 0},
  {384, 48, 3, {6,8,8}, 512, (const void*)&axis_pass_static<double,512,384,48,6,8,8>, (const void*)&axis_pass_any<double,512,false,384,48,6,8,8>, (const void*)&axis_pass_pipe<double,512,false,8,384,48,6,8,8>, (const void*)&axis_pass_pipe<double,512,true,0,384,48,6,8,8>, 512, 8},
  {405, 27, 4, {15,3,3,3}, 512, (const void*)&axis_pass_static<double,512,405,27,15,3,3,3>, (const void*)&axis_pass_any<double,512,false,405,27,15,3,3,3>, (const void*)&axis_pass_pipe<double,512,false,8,405,27,15,3,3,3>, (const void*)&axis_pass_pipe<double,512,true,0,405,27,15,3,3,3>, 512, 8},
  {441, 63, 4, {7,7,3,3}, 512, (const void*)&axis_pass_static<double,512,441,63,7,7,3,3>, (const void*)&axis_pass_any<double,512,false,441,63,7,7,3,3>, nullptr, nullptr, 512, 0},
  {480, 48, 3, {10,6,8}, 512, (const void*)&axis_pass_static<double,512,480,48,10,6,8>, (const void*)&axis_pass_any<double,512,false,480,48,10,6,8>, (const void*)&axis_pass_pipe<double,512,false,8,480,48,10,6,8>, (const void*)&axis_pass_pipe<double,512,true,0,480,48,10,6,8>, 512, 8},
  {504, 42, 3, {12,7,6}, 512, (const void*)&axis_pass_static<double,512,504,42,12,7,6>, (const void*)&axis_pass_any<double,512,false,504,42,12,7,6>, nullptr, nullptr, 512, 0},
  {539, 49, 3, {11,7,7}, 512, (const void*)&axis_pass_static<double,512,539,49,11,7,7>, (const void*)&axis_pass_any<double,512,false,539,49,11,7,7>, nullptr, nullptr, 512, 0},
  {572, 44, 3, {13,11,4}, 512, (const void*)&axis_pass_static<double,512,572,44,13,11,4>, (const void*)&axis_pass_any<double,512,false,572,44,13,11,4>, nullptr, nullptr, 512, 0},
  {605, 55, 3, {11,11,5}, 512, (const void*)&axis_pass_static<double,512,605,55,11,11,5>, (const void*)&axis_pass_any<double,512,false,605,55,11,11,5>, nullptr, nullptr, 512, 0},
  {640, 64, 3, {10,8,8}, 512, (const void*)&axis_pass_static<double,512,640,64,10,8,8>, (const void*)&axis_pass_any<double,512,false,640,64,10,8,8>, nullptr, nullptr, 512, 0},
  {676, 52, 3, {13,13,4}, 512, (const void*)&axis_pass_static<double,512,676,52,13,13,4>, (const void*)&axis_pass_any<double,512,false,676,52,13,13,4>, nullptr, nullptr, 512, 0},
  {715, 55, 3, {13,11,5}, 512, (const void*)&axis_pass_static<double,512,715,55,13,11,5>, (const void*)&axis_pass_any<double,512,false,715,55,13,11,5>, nullptr, nullptr, 512, 0},
  {750, 50, 3, {15,10,5}, 512, (const void*)&axis_pass_static<double,512,750,50,15,10,5>, (const void*)&axis_pass_any<double,512,false,750,50,15,10,5>, nullptr, nullptr, 512, 0},
  {792, 66, 3, {12,11,6}, 512, (const void*)&axis_pass_static<double,512,792,66,12,11,6>, (const void*)&axis_pass_any<double,512,false,792,66,12,11,6>, nullptr, nullptr, 512, 0},
  {840, 70, 3, {12,10,7}, 512, (const void*)&axis_pass_static<double,512,840,70,12,10,7>, (const void*)&axis_pass_any<double,512,false,840,70,12,10,7>, nullptr, nullptr, 512, 0},
  {880, 80, 3, {11,10,8}, 512, (const void*)&axis_pass_static<double,512,880,80,11,10,8>, (const void*)&axis_pass_any<double,512,false,880,80,11,10,8>, nullptr, nullptr, 512, 0},
  {924, 77, 3, {12,11,7}, 512, (const void*)&axis_pass_static<double,512,924,77,12,11,7>, (const void*)&axis_pass_any<double,512,false,924,77,12,11,7>, nullptr, nullptr, 512, 0},
  {975, 65, 3, {15,13,5}, 256, (const void*)&axis_pass_static<double,256,975,65,15,13,5>, (const void*)&axis_pass_any<double,256,false,975,65,15,13,5>, nullptr, nullptr, 256, 0},
  {1014, 78, 3, {13,13,6}, 512, (const void*)&axis_pass_static<double,512,1014,78,13,13,6>, (const void*)&axis_pass_any<double,512,false,1014,78,13,13,6>, nullptr, nullptr, 512, 0},
  {1215, 81, 5, {15,3,3,3,3}, 512, (const void*)&axis_pass_static<double,512,1215,81,15,3,3,3,3>, (const void*)&axis_pass_any<double,512,false,1215,81,15,3,3,3,3>, nullptr, nullptr, 512, 0},
  {1458, 243, 6, {6,3,3,3,3,3}, 1024, (const void*)&axis_pass_static<double,1024,1458,243,6,3,3,3,3,3>, (const void*)&axis_pass_any<double,1024,false,1458,243,6,3,3,3,3,3>, nullptr, nullptr, 512, 0},
  {1800, 120, 3, {15,12,10}, 512, (const void*)&axis_pass_static<double,512,1800,120,15,12,10>, (const void*)&axis_pass_any<double,512,false,1800,120,15,12,10>, nullptr, nullptr, 512, 0},
  {2048, 128, 3, {16,16,8}, 512, (const void*)&axis_pass_static<double,512,2048,128,16,16,8>, (const void*)&axis_pass_any<double,512,false,2048,128,16,16,8>, nullptr, nullptr, 512, 0},
};
const int kPlansCount_f64_4 = 45;
}  // namespace dfft
