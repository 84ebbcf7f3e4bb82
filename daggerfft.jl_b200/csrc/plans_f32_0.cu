// Generated by gen_plans.py -- do not edit.
#include "static_plans.h"
namespace dfft {
template __global__ void axis_pass_static<float,1024,1,1,1>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,1,1,1>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,7,1,7>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,7,1,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,13,1,13>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,13,1,13>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,21,3,7,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,21,3,7,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,28,4,7,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,28,4,7,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,39,3,13,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,39,3,13,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,49,7,7,7>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,49,7,7,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,60,6,10,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,60,6,10,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,60,6,10,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,60,6,10,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,72,6,12,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,72,6,12,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,72,6,12,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,72,6,12,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,84,7,12,7>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,84,7,12,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,99,9,11,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,99,9,11,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,112,8,14,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,112,8,14,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,128,8,16,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,128,8,16,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,128,8,16,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,128,8,16,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,144,12,12,12>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,144,12,12,12>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,144,12,12,12>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,144,12,12,12>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,162,27,6,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,162,27,6,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,162,27,6,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,162,27,6,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,180,12,15,12>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,180,12,15,12>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,16,180,12,15,12>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,180,12,15,12>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,198,18,11,6,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,198,18,11,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,224,14,14,16>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,224,14,14,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,243,81,3,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,243,81,3,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,8,243,81,3,3,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,243,81,3,3,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,264,24,11,6,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,264,24,11,6,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,288,36,6,6,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,288,36,6,6,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,288,36,6,6,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,288,36,6,6,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,315,21,15,7,3>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,315,21,15,7,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,338,26,13,13,2>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,338,26,13,13,2>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,363,33,11,11,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,363,33,11,11,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,390,30,13,6,5>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,390,30,13,6,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,420,42,10,7,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,420,42,10,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,450,30,15,6,5>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,450,30,15,6,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,16,450,30,15,6,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,450,30,15,6,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,486,81,6,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,486,81,6,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,8,486,81,6,3,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,486,81,6,3,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,512,64,8,8,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,512,64,8,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,512,64,8,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,512,64,8,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,546,42,13,7,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,546,42,13,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,585,39,15,13,3>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,585,39,15,13,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,624,48,13,6,8>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,624,48,13,6,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,650,50,13,10,5>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,650,50,13,10,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,693,63,11,7,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,693,63,11,7,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,726,66,11,11,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,726,66,11,11,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,768,64,12,8,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,768,64,12,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,8,768,64,12,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,768,64,12,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,810,54,15,6,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,810,54,15,6,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,8,810,54,15,6,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,810,54,15,6,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,847,77,11,11,7>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,847,77,11,11,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,891,81,11,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,891,81,11,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,945,63,15,7,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,945,63,15,7,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,990,66,15,11,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,990,66,15,11,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,1080,72,15,12,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,1080,72,15,12,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,1280,80,10,16,8>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,1280,80,10,16,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,1536,96,12,16,8>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,1536,96,12,16,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,1920,120,12,10,16>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,1920,120,12,10,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,2187,729,3,3,3,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,2187,729,3,3,3,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,2560,160,10,16,16>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,2560,160,10,16,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,3072,192,12,16,16>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,3072,192,12,16,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,3600,225,15,15,16>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,3600,225,15,15,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,4050,270,15,15,6,3>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,4050,270,15,15,6,3>(const __grid_constant__ PassDesc);
extern const StaticPlan kPlans_f32_0[];
extern const int kPlansCount_f32_0;
const StaticPlan kPlans_f32_0[] = {
  {1, 1, 1, {1}, 1024, (const void*)&axis_pass_static<float,1024,1,1,1>, (const void*)&axis_pass_any<float,1024,false,1,1,1>, nullptr, nullptr, 1024, 0},
  {7, 1, 1, {7}, 1024, (const void*)&axis_pass_static<float,1024,7,1,7>, (const void*)&axis_pass_any<float,1024,false,7,1,7>, nullptr, nullptr, 1024, 0},
  {13, 1, 1, {13}, 1024, (const void*)&axis_pass_static<float,1024,13,1,13>, (const void*)&axis_pass_any<float,1024,false,13,1,13>, nullptr, nullptr, 1024, 0},
  {21, 3, 2, {7,3}, 1024, (const void*)&axis_pass_static<float,1024,21,3,7,3>, (const void*)&axis_pass_any<float,1024,false,21,3,7,3>, nullptr, nullptr, 1024, 0},
  {28, 4, 2, {7,4}, 1024, (const void*)&axis_pass_static<float,1024,28,4,7,4>, (const void*)&axis_pass_any<float,1024,false,28,4,7,4>, nullptr, nullptr, 1024, 0},
  {39, 3, 2, {13,3}, 1024, (const void*)&axis_pass_static<float,1024,39,3,13,3>, (const void*)&axis_pass_any<float,1024,false,39,3,13,3>, nullptr, nullptr, 1024, 0},
  {49, 7, 2, {7,7}, 1024, (const void*)&axis_pass_static<float,1024,49,7,7,7>, (const void*)&axis_pass_any<float,1024,false,49,7,7,7>, nullptr, nullptr, 1024, 0},
  {60, 6, 2, {10,6}, 1024, (const void*)&axis_pass_static<float,1024,60,6,10,6>, (const void*)&axis_pass_any<float,1024,false,60,6,10,6>, (const void*)&axis_pass_pipe<float,1024,false,16,60,6,10,6>, (const void*)&axis_pass_pipe<float,1024,true,0,60,6,10,6>, 1024, 16},
  {72, 6, 2, {12,6}, 1024, (const void*)&axis_pass_static<float,1024,72,6,12,6>, (const void*)&axis_pass_any<float,1024,false,72,6,12,6>, (const void*)&axis_pass_pipe<float,1024,false,16,72,6,12,6>, (const void*)&axis_pass_pipe<float,1024,true,0,72,6,12,6>, 1024, 16},
  {84, 7, 2, {12,7}, 1024, (const void*)&axis_pass_static<float,1024,84,7,12,7>, (const void*)&axis_pass_any<float,1024,false,84,7,12,7>, nullptr, nullptr, 1024, 0},
  {99, 9, 3, {11,3,3}, 1024, (const void*)&axis_pass_static<float,1024,99,9,11,3,3>, (const void*)&axis_pass_any<float,1024,false,99,9,11,3,3>, nullptr, nullptr, 1024, 0},
  {112, 8, 2, {14,8}, 1024, (const void*)&axis_pass_static<float,1024,112,8,14,8>, (const void*)&axis_pass_any<float,1024,false,112,8,14,8>, nullptr, nullptr, 1024, 0},
  {128, 8, 2, {16,8}, 1024, (const void*)&axis_pass_static<float,1024,128,8,16,8>, (const void*)&axis_pass_any<float,1024,false,128,8,16,8>, (const void*)&axis_pass_pipe<float,1024,false,16,128,8,16,8>, (const void*)&axis_pass_pipe<float,1024,true,0,128,8,16,8>, 1024, 16},
  {144, 12, 2, {12,12}, 1024, (const void*)&axis_pass_static<float,1024,144,12,12,12>, (const void*)&axis_pass_any<float,1024,false,144,12,12,12>, (const void*)&axis_pass_pipe<float,1024,false,16,144,12,12,12>, (const void*)&axis_pass_pipe<float,1024,true,0,144,12,12,12>, 1024, 16},
  {162, 27, 4, {6,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,162,27,6,3,3,3>, (const void*)&axis_pass_any<float,1024,false,162,27,6,3,3,3>, (const void*)&axis_pass_pipe<float,1024,false,16,162,27,6,3,3,3>, (const void*)&axis_pass_pipe<float,1024,true,0,162,27,6,3,3,3>, 1024, 16},
  {180, 12, 2, {15,12}, 512, (const void*)&axis_pass_static<float,512,180,12,15,12>, (const void*)&axis_pass_any<float,512,false,180,12,15,12>, (const void*)&axis_pass_pipe<float,512,false,16,180,12,15,12>, (const void*)&axis_pass_pipe<float,512,true,0,180,12,15,12>, 512, 16},
  {198, 18, 3, {11,6,3}, 1024, (const void*)&axis_pass_static<float,1024,198,18,11,6,3>, (const void*)&axis_pass_any<float,1024,false,198,18,11,6,3>, nullptr, nullptr, 1024, 0},
  {224, 14, 2, {14,16}, 512, (const void*)&axis_pass_static<float,512,224,14,14,16>, (const void*)&axis_pass_any<float,512,false,224,14,14,16>, nullptr, nullptr, 512, 0},
  {243, 81, 5, {3,3,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,243,81,3,3,3,3,3>, (const void*)&axis_pass_any<float,1024,false,243,81,3,3,3,3,3>, (const void*)&axis_pass_pipe<float,1024,false,8,243,81,3,3,3,3,3>, (const void*)&axis_pass_pipe<float,1024,true,0,243,81,3,3,3,3,3>, 1024, 8},
  {264, 24, 3, {11,6,4}, 1024, (const void*)&axis_pass_static<float,1024,264,24,11,6,4>, (const void*)&axis_pass_any<float,1024,false,264,24,11,6,4>, nullptr, nullptr, 1024, 0},
  {288, 36, 3, {6,6,8}, 1024, (const void*)&axis_pass_static<float,1024,288,36,6,6,8>, (const void*)&axis_pass_any<float,1024,false,288,36,6,6,8>, (const void*)&axis_pass_pipe<float,1024,false,16,288,36,6,6,8>, (const void*)&axis_pass_pipe<float,1024,true,0,288,36,6,6,8>, 1024, 16},
  {315, 21, 3, {15,7,3}, 512, (const void*)&axis_pass_static<float,512,315,21,15,7,3>, (const void*)&axis_pass_any<float,512,false,315,21,15,7,3>, nullptr, nullptr, 512, 0},
  {338, 26, 3, {13,13,2}, 1024, (const void*)&axis_pass_static<float,1024,338,26,13,13,2>, (const void*)&axis_pass_any<float,1024,false,338,26,13,13,2>, nullptr, nullptr, 1024, 0},
  {363, 33, 3, {11,11,3}, 1024, (const void*)&axis_pass_static<float,1024,363,33,11,11,3>, (const void*)&axis_pass_any<float,1024,false,363,33,11,11,3>, nullptr, nullptr, 1024, 0},
  {390, 30, 3, {13,6,5}, 512, (const void*)&axis_pass_static<float,512,390,30,13,6,5>, (const void*)&axis_pass_any<float,512,false,390,30,13,6,5>, nullptr, nullptr, 512, 0},
  {420, 42, 3, {10,7,6}, 1024, (const void*)&axis_pass_static<float,1024,420,42,10,7,6>, (const void*)&axis_pass_any<float,1024,false,420,42,10,7,6>, nullptr, nullptr, 1024, 0},
  {450, 30, 3, {15,6,5}, 512, (const void*)&axis_pass_static<float,512,450,30,15,6,5>, (const void*)&axis_pass_any<float,512,false,450,30,15,6,5>, (const void*)&axis_pass_pipe<float,512,false,16,450,30,15,6,5>, (const void*)&axis_pass_pipe<float,512,true,0,450,30,15,6,5>, 512, 16},
  {486, 81, 5, {6,3,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,486,81,6,3,3,3,3>, (const void*)&axis_pass_any<float,1024,false,486,81,6,3,3,3,3>, (const void*)&axis_pass_pipe<float,1024,false,8,486,81,6,3,3,3,3>, (const void*)&axis_pass_pipe<float,1024,true,0,486,81,6,3,3,3,3>, 1024, 8},
  {512, 64, 3, {8,8,8}, 1024, (const void*)&axis_pass_static<float,1024,512,64,8,8,8>, (const void*)&axis_pass_any<float,1024,false,512,64,8,8,8>, (const void*)&axis_pass_pipe<float,1024,false,16,512,64,8,8,8>, (const void*)&axis_pass_pipe<float,1024,true,0,512,64,8,8,8>, 1024, 16},
  {546, 42, 3, {13,7,6}, 512, (const void*)&axis_pass_static<float,512,546,42,13,7,6>, (const void*)&axis_pass_any<float,512,false,546,42,13,7,6>, nullptr, nullptr, 512, 0},
  {585, 39, 3, {15,13,3}, 512, (const void*)&axis_pass_static<float,512,585,39,15,13,3>, (const void*)&axis_pass_any<float,512,false,585,39,15,13,3>, nullptr, nullptr, 512, 0},
  {624, 48, 3, {13,6,8}, 512, (const void*)&axis_pass_static<float,512,624,48,13,6,8>, (const void*)&axis_pass_any<float,512,false,624,48,13,6,8>, nullptr, nullptr, 512, 0},
  {650, 50, 3, {13,10,5}, 512, (const void*)&axis_pass_static<float,512,650,50,13,10,5>, (const void*)&axis_pass_any<float,512,false,650,50,13,10,5>, nullptr, nullptr, 512, 0},
  {693, 63, 4, {11,7,3,3}, 1024, (const void*)&axis_pass_static<float,1024,693,63,11,7,3,3>, (const void*)&axis_pass_any<float,1024,false,693,63,11,7,3,3>, nullptr, nullptr, 1024, 0},
  {726, 66, 3, {11,11,6}, 1024, (const void*)&axis_pass_static<float,1024,726,66,11,11,6>, (const void*)&axis_pass_any<float,1024,false,726,66,11,11,6>, nullptr, nullptr, 1024, 0},
  {768, 64, 3, {12,8,8}, 1024, (const void*)&axis_pass_static<float,1024,768,64,12,8,8>, (const void*)&axis_pass_any<float,1024,false,768,64,12,8,8>, (const void*)&axis_pass_pipe<float,1024,false,8,768,64,12,8,8>, (const void*)&axis_pass_pipe<float,1024,true,0,768,64,12,8,8>, 1024, 8},
  {810, 54, 4, {15,6,3,3}, 512, (const void*)&axis_pass_static<float,512,810,54,15,6,3,3>, (const void*)&axis_pass_any<float,512,false,810,54,15,6,3,3>, (const void*)&axis_pass_pipe<float,512,false,8,810,54,15,6,3,3>, (const void*)&axis_pass_pipe<float,512,true,0,810,54,15,6,3,3>, 512, 8},
  {847, 77, 3, {11,11,7}, 1024, (const void*)&axis_pass_static<float,1024,847,77,11,11,7>, (const void*)&axis_pass_any<float,1024,false,847,77,11,11,7>, nullptr, nullptr, 1024, 0},
  {891, 81, 5, {11,3,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,891,81,11,3,3,3,3>, (const void*)&axis_pass_any<float,1024,false,891,81,11,3,3,3,3>, nullptr, nullptr, 1024, 0},
  {945, 63, 4, {15,7,3,3}, 512, (const void*)&axis_pass_static<float,512,945,63,15,7,3,3>, (const void*)&axis_pass_any<float,512,false,945,63,15,7,3,3>, nullptr, nullptr, 512, 0},
  {990, 66, 3, {15,11,6}, 512, (const void*)&axis_pass_static<float,512,990,66,15,11,6>, (const void*)&axis_pass_any<float,512,false,990,66,15,11,6>, nullptr, nullptr, 512, 0},
  {1080, 72, 3, {15,12,6}, 512, (const void*)&axis_pass_static<float,512,1080,72,15,12,6>, (const void*)&axis_pass_any<float,512,false,1080,72,15,12,6>, nullptr, nullptr, 512, 0},
  {1280, 80, 3, {10,16,8}, 512, (const void*)&axis_pass_static<float,512,1280,80,10,16,8>, (const void*)&axis_pass_any<float,512,false,1280,80,10,16,8>, nullptr, nullptr, 512, 0},
  {1536, 96, 3, {12,16,8}, 512, (const void*)&axis_pass_static<float,512,1536,96,12,16,8>, (const void*)&axis_pass_any<float,512,false,1536,96,12,16,8>, nullptr, nullptr, 512, 0},
  {1920, 120, 3, {12,10,16}, 512, (const void*)&axis_pass_static<float,512,1920,120,12,10,16>, (const void*)&axis_pass_any<float,512,false,1920,120,12,10,16>, nullptr, nullptr, 512, 0},
  {2187, 729, 7, {3,3,3,3,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,2187,729,3,3,3,3,3,3,3>, (const void*)&axis_pass_any<float,1024,false,2187,729,3,3,3,3,3,3,3>, nullptr, nullptr, 1024, 0},
  {2560, 160, 3, {10,16,16}, 512, (const void*)&axis_pass_static<float,512,2560,160,10,16,16>, (const void*)&axis_pass_any<float,512,false,2560,160,10,16,16>, nullptr, nullptr, 512, 0},
  {3072, 192, 3, {12,16,16}, 512, (const void*)&axis_pass_static<float,512,3072,192,12,16,16>, (const void*)&axis_pass_any<float,512,false,3072,192,12,16,16>, nullptr, nullptr, 512, 0},
  {3600, 225, 3, {15,15,16}, 512, (const void*)&axis_pass_static<float,512,3600,225,15,15,16>, (const void*)&axis_pass_any<float,512,false,3600,225,15,15,16>, nullptr, nullptr, 512, 0},
  {4050, 270, 4, {15,15,6,3}, 512, (const void*)&axis_pass_static<float,512,4050,270,15,15,6,3>, (const void*)&axis_pass_any<float,512,false,4050,270,15,15,6,3>, nullptr, nullptr, 512, 0},
};
const int kPlansCount_f32_0 = 50;
}  // namespace dfft
