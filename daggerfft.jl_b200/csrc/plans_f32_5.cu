// Generated by gen_plans.py -- do not edit.
#include "static_plans.h"
namespace dfft {
template __global__ void axis_pass_static<float,1024,6,1,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,6,1,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,12,1,12>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,12,1,12>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,12,1,12>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,12,1,12>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,20,4,5,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,20,4,5,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,20,4,5,4>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,20,4,5,4>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,27,9,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,27,9,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,27,9,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,27,9,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,36,6,6,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,36,6,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,36,6,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,36,6,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,48,6,6,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,48,6,6,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,48,6,6,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,48,6,6,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,56,7,7,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,56,7,7,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,70,7,10,7>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,70,7,10,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,81,27,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,81,27,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,81,27,3,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,81,27,3,3,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,98,7,14,7>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,98,7,14,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,110,10,11,10>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,110,10,11,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,126,18,7,6,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,126,18,7,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,143,11,13,11>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,143,11,13,11>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,160,10,10,16>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,160,10,10,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,16,160,10,10,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,160,10,10,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,512,176,11,11,16>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,176,11,11,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,196,14,14,14>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,196,14,14,14>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,220,20,11,5,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,220,20,11,5,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,242,22,11,11,2>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,242,22,11,11,2>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,260,20,13,5,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,260,20,13,5,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,286,22,13,11,2>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,286,22,13,11,2>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,312,24,13,6,4>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,312,24,13,6,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,336,42,7,6,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,336,42,7,6,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,360,36,10,6,6>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,360,36,10,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,360,36,10,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,360,36,10,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,385,35,11,7,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,385,35,11,7,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,416,32,13,8,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,416,32,13,8,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,448,56,7,8,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,448,56,7,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,484,44,11,11,4>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,484,44,11,11,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,507,39,13,13,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,507,39,13,13,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,540,36,15,6,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,540,36,15,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,8,540,36,15,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,540,36,15,6,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,576,48,12,6,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,576,48,12,6,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,16,576,48,12,6,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,576,48,12,6,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,616,56,11,7,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,616,56,11,7,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,648,108,6,6,6,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,648,108,6,6,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,8,648,108,6,6,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,648,108,6,6,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,686,49,14,7,7>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,686,49,14,7,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,720,60,12,10,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,720,60,12,10,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,512,false,8,720,60,12,10,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,512,true,0,720,60,12,10,6>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,756,108,7,6,6,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,756,108,7,6,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,800,80,10,10,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,800,80,10,10,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,8,800,80,10,10,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,800,80,10,10,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,845,65,13,13,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,845,65,13,13,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,882,126,7,7,6,3>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,882,126,7,7,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,936,72,13,12,6>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,936,72,13,12,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,980,70,14,10,7>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,980,70,14,10,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,1024,64,16,8,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,1024,64,16,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<float,1024,false,8,1024,64,16,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<float,1024,true,0,1024,64,16,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<float,1024,1250,125,10,5,5,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,1250,125,10,5,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,1500,100,15,10,10>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,1500,100,15,10,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,1875,125,15,5,5,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,1875,125,15,5,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,512,2160,144,15,12,12>(const PassDesc);
template __global__ void axis_pass_any<float,512,false,2160,144,15,12,12>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,2500,250,10,10,5,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,2500,250,10,10,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,3000,300,10,10,6,5>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,3000,300,10,10,6,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,3456,288,12,6,6,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,3456,288,12,6,6,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<float,1024,4000,400,10,10,5,8>(const PassDesc);
template __global__ void axis_pass_any<float,1024,false,4000,400,10,10,5,8>(const __grid_constant__ PassDesc);
extern const StaticPlan kPlans_f32_5[];
extern const int kPlansCount_f32_5;
const StaticPlan kPlans_f32_5[] = {
  {6, 1, 1, {6}, 1024, (const void*)&axis_pass_static<float,1024,6,1,6>, (const void*)&axis_pass_any<float,1024,false,6,1,6>, nullptr, nullptr, 1024, 0},
  {12, 1, 1, {12}, 1024, (const void*)&axis_pass_static<float,1024,12,1,12>, (const void*)&axis_pass_any<float,1024,false,12,1,12>, (const void*)&axis_pass_pipe<float,1024,false,16,12,1,12>, (const void*)&axis_pass_pipe<float,1024,true,0,12,1,12>, 1024, 16},
  {20, 4, 2, {5,4}, 1024, (const void*)&axis_pass_static<float,1024,20,4,5,4>, (const void*)&axis_pass_any<float,1024,false,20,4,5,4>, (const void*)&axis_pass_pipe<float,1024,false,16,20,4,5,4>, (const void*)&axis_pass_pipe<float,1024,true,0,20,4,5,4>, 1024, 16},
  {27, 9, 3, {3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,27,9,3,3,3>, (const void*)&axis_pass_any<float,1024,false,27,9,3,3,3>, (const void*)&axis_pass_pipe<float,1024,false,16,27,9,3,3,3>, (const void*)&axis_pass_pipe<float,1024,true,0,27,9,3,3,3>, 1024, 16},
  {36, 6, 2, {6,6}, 1024, (const void*)&axis_pass_static<float,1024,36,6,6,6>, (const void*)&axis_pass_any<float,1024,false,36,6,6,6>, (const void*)&axis_pass_pipe<float,1024,false,16,36,6,6,6>, (const void*)&axis_pass_pipe<float,1024,true,0,36,6,6,6>, 1024, 16},
  {48, 6, 2, {6,8}, 1024, (const void*)&axis_pass_static<float,1024,48,6,6,8>, (const void*)&axis_pass_any<float,1024,false,48,6,6,8>, (const void*)&axis_pass_pipe<float,1024,false,16,48,6,6,8>, (const void*)&axis_pass_pipe<float,1024,true,0,48,6,6,8>, 1024, 16},
  {56, 7, 2, {7,8}, 1024, (const void*)&axis_pass_static<float,1024,56,7,7,8>, (const void*)&axis_pass_any<float,1024,false,56,7,7,8>, nullptr, nullptr, 1024, 0},
  {70, 7, 2, {10,7}, 1024, (const void*)&axis_pass_static<float,1024,70,7,10,7>, (const void*)&axis_pass_any<float,1024,false,70,7,10,7>, nullptr, nullptr, 1024, 0},
  {81, 27, 4, {3,3,3,3}, 1024, (const void*)&axis_pass_static<float,1024,81,27,3,3,3,3>, (const void*)&axis_pass_any<float,1024,false,81,27,3,3,3,3>, (const void*)&axis_pass_pipe<float,1024,false,16,81,27,3,3,3,3>, (const void*)&axis_pass_pipe<float,1024,true,0,81,27,3,3,3,3>, 1024, 16},
  {98, 7, 2, {14,7}, 1024, (const void*)&axis_pass_static<float,1024,98,7,14,7>, (const void*)&axis_pass_any<float,1024,false,98,7,14,7>, nullptr, nullptr, 1024, 0},
  {110, 10, 2, {11,10}, 512, (const void*)&axis_pass_static<float,512,110,10,11,10>, (const void*)&axis_pass_any<float,512,false,110,10,11,10>, nullptr, nullptr, 512, 0},
  {126, 18, 3, {7,6,3}, 1024, (const void*)&axis_pass_static<float,1024,126,18,7,6,3>, (const void*)&axis_pass_any<float,1024,false,126,18,7,6,3>, nullptr, nullptr, 1024, 0},
  {143, 11, 2, {13,11}, 512, (const void*)&axis_pass_static<float,512,143,11,13,11>, (const void*)&axis_pass_any<float,512,false,143,11,13,11>, nullptr, nullptr, 512, 0},
  {160, 10, 2, {10,16}, 512, (const void*)&axis_pass_static<float,512,160,10,10,16>, (const void*)&axis_pass_any<float,512,false,160,10,10,16>, (const void*)&axis_pass_pipe<float,512,false,16,160,10,10,16>, (const void*)&axis_pass_pipe<float,512,true,0,160,10,10,16>, 512, 16},
  {176, 11, 2, {11,16}, 512, (const void*)&axis_pass_static<float,512,176,11,11,16>, (const void*)&axis_pass_any<float,512,false,176,11,11,16>, nullptr, nullptr, 512, 0},
  {196, 14, 2, {14,14}, 1024, (const void*)&axis_pass_static<float,1024,196,14,14,14>, (const void*)&axis_pass_any<float,1024,false,196,14,14,14>, nullptr, nullptr, 1024, 0},
  {220, 20, 3, {11,5,4}, 1024, (const void*)&axis_pass_static<float,1024,220,20,11,5,4>, (const void*)&axis_pass_any<float,1024,false,220,20,11,5,4>, nullptr, nullptr, 1024, 0},
  {242, 22, 3, {11,11,2}, 1024, (const void*)&axis_pass_static<float,1024,242,22,11,11,2>, (const void*)&axis_pass_any<float,1024,false,242,22,11,11,2>, nullptr, nullptr, 1024, 0},
  {260, 20, 3, {13,5,4}, 1024, (const void*)&axis_pass_static<float,1024,260,20,13,5,4>, (const void*)&axis_pass_any<float,1024,false,260,20,13,5,4>, nullptr, nullptr, 1024, 0},
  {286, 22, 3, {13,11,2}, 512, (const void*)&axis_pass_static<float,512,286,22,13,11,2>, (const void*)&axis_pass_any<float,512,false,286,22,13,11,2>, nullptr, nullptr, 512, 0},
  {312, 24, 3, {13,6,4}, 512, (const void*)&axis_pass_static<float,512,312,24,13,6,4>, (const void*)&axis_pass_any<float,512,false,312,24,13,6,4>, nullptr, nullptr, 512, 0},
  {336, 42, 3, {7,6,8}, 1024, (const void*)&axis_pass_static<float,1024,336,42,7,6,8>, (const void*)&axis_pass_any<float,1024,false,336,42,7,6,8>, nullptr, nullptr, 1024, 0},
  {360, 36, 3, {10,6,6}, 1024, (const void*)&axis_pass_static<float,1024,360,36,10,6,6>, (const void*)&axis_pass_any<float,1024,false,360,36,10,6,6>, (const void*)&axis_pass_pipe<float,1024,false,16,360,36,10,6,6>, (const void*)&axis_pass_pipe<float,1024,true,0,360,36,10,6,6>, 1024, 16},
  {385, 35, 3, {11,7,5}, 1024, (const void*)&axis_pass_static<float,1024,385,35,11,7,5>, (const void*)&axis_pass_any<float,1024,false,385,35,11,7,5>, nullptr, nullptr, 1024, 0},
  {416, 32, 3, {13,8,4}, 1024, (const void*)&axis_pass_static<float,1024,416,32,13,8,4>, (const void*)&axis_pass_any<float,1024,false,416,32,13,8,4>, nullptr, nullptr, 1024, 0},
  {448, 56, 3, {7,8,8}, 1024, (const void*)&axis_pass_static<float,1024,448,56,7,8,8>, (const void*)&axis_pass_any<float,1024,false,448,56,7,8,8>, nullptr, nullptr, 1024, 0},
  {484, 44, 3, {11,11,4}, 1024, (const void*)&axis_pass_static<float,1024,484,44,11,11,4>, (const void*)&axis_pass_any<float,1024,false,484,44,11,11,4>, nullptr, nullptr, 1024, 0},
  {507, 39, 3, {13,13,3}, 1024, (const void*)&axis_pass_static<float,1024,507,39,13,13,3>, (const void*)&axis_pass_any<float,1024,false,507,39,13,13,3>, nullptr, nullptr, 1024, 0},
  {540, 36, 3, {15,6,6}, 512, (const void*)&axis_pass_static<float,512,540,36,15,6,6>, (const void*)&axis_pass_any<float,512,false,540,36,15,6,6>, (const void*)&axis_pass_pipe<float,512,false,8,540,36,15,6,6>, (const void*)&axis_pass_pipe<float,512,true,0,540,36,15,6,6>, 512, 8},
  {576, 48, 3, {12,6,8}, 1024, (const void*)&axis_pass_static<float,1024,576,48,12,6,8>, (const void*)&axis_pass_any<float,1024,false,576,48,12,6,8>, (const void*)&axis_pass_pipe<float,1024,false,16,576,48,12,6,8>, (const void*)&axis_pass_pipe<float,1024,true,0,576,48,12,6,8>, 1024, 16},
  {616, 56, 3, {11,7,8}, 1024, (const void*)&axis_pass_static<float,1024,616,56,11,7,8>, (const void*)&axis_pass_any<float,1024,false,616,56,11,7,8>, nullptr, nullptr, 1024, 0},
  {648, 108, 4, {6,6,6,3}, 1024, (const void*)&axis_pass_static<float,1024,648,108,6,6,6,3>, (const void*)&axis_pass_any<float,1024,false,648,108,6,6,6,3>, (const void*)&axis_pass_pipe<float,1024,false,8,648,108,6,6,6,3>, (const void*)&axis_pass_pipe<float,1024,true,0,648,108,6,6,6,3>, 1024, 8},
  {686, 49, 3, {14,7,7}, 1024, (const void*)&axis_pass_static<float,1024,686,49,14,7,7>, (const void*)&axis_pass_any<float,1024,false,686,49,14,7,7>, nullptr, nullptr, 1024, 0},
  {720, 60, 3, {12,10,6}, 512, (const void*)&axis_pass_static<float,512,720,60,12,10,6>, (const void*)&axis_pass_any<float,512,false,720,60,12,10,6>, (const void*)&axis_pass_pipe<float,512,false,8,720,60,12,10,6>, (const void*)&axis_pass_pipe<float,512,true,0,720,60,12,10,6>, 512, 8},
  {756, 108, 4, {7,6,6,3}, 1024, (const void*)&axis_pass_static<float,1024,756,108,7,6,6,3>, (const void*)&axis_pass_any<float,1024,false,756,108,7,6,6,3>, nullptr, nullptr, 1024, 0},
  {800, 80, 3, {10,10,8}, 1024, (const void*)&axis_pass_static<float,1024,800,80,10,10,8>, (const void*)&axis_pass_any<float,1024,false,800,80,10,10,8>, (const void*)&axis_pass_pipe<float,1024,false,8,800,80,10,10,8>, (const void*)&axis_pass_pipe<float,1024,true,0,800,80,10,10,8>, 1024, 8},
  {845, 65, 3, {13,13,5}, 1024, (const void*)&axis_pass_static<float,1024,845,65,13,13,5>, (const void*)&axis_pass_any<float,1024,false,845,65,13,13,5>, nullptr, nullptr, 1024, 0},
  {882, 126, 4, {7,7,6,3}, 1024, (const void*)&axis_pass_static<float,1024,882,126,7,7,6,3>, (const void*)&axis_pass_any<float,1024,false,882,126,7,7,6,3>, nullptr, nullptr, 1024, 0},
  {936, 72, 3, {13,12,6}, 512, (const void*)&axis_pass_static<float,512,936,72,13,12,6>, (const void*)&axis_pass_any<float,512,false,936,72,13,12,6>, nullptr, nullptr, 512, 0},
  {980, 70, 3, {14,10,7}, 512, (const void*)&axis_pass_static<float,512,980,70,14,10,7>, (const void*)&axis_pass_any<float,512,false,980,70,14,10,7>, nullptr, nullptr, 512, 0},
  {1024, 64, 3, {16,8,8}, 1024, (const void*)&axis_pass_static<float,1024,1024,64,16,8,8>, (const void*)&axis_pass_any<float,1024,false,1024,64,16,8,8>, (const void*)&axis_pass_pipe<float,1024,false,8,1024,64,16,8,8>, (const void*)&axis_pass_pipe<float,1024,true,0,1024,64,16,8,8>, 1024, 8},
  {1250, 125, 4, {10,5,5,5}, 1024, (const void*)&axis_pass_static<float,1024,1250,125,10,5,5,5>, (const void*)&axis_pass_any<float,1024,false,1250,125,10,5,5,5>, nullptr, nullptr, 1024, 0},
  {1500, 100, 3, {15,10,10}, 512, (const void*)&axis_pass_static<float,512,1500,100,15,10,10>, (const void*)&axis_pass_any<float,512,false,1500,100,15,10,10>, nullptr, nullptr, 512, 0},
  {1875, 125, 4, {15,5,5,5}, 1024, (const void*)&axis_pass_static<float,1024,1875,125,15,5,5,5>, (const void*)&axis_pass_any<float,1024,false,1875,125,15,5,5,5>, nullptr, nullptr, 1024, 0},
  {2160, 144, 3, {15,12,12}, 512, (const void*)&axis_pass_static<float,512,2160,144,15,12,12>, (const void*)&axis_pass_any<float,512,false,2160,144,15,12,12>, nullptr, nullptr, 512, 0},
  {2500, 250, 4, {10,10,5,5}, 1024, (const void*)&axis_pass_static<float,1024,2500,250,10,10,5,5>, (const void*)&axis_pass_any<float,1024,false,2500,250,10,10,5,5>, nullptr, nullptr, 1024, 0},
  {3000, 300, 4, {10,10,6,5}, 1024, (const void*)&axis_pass_static<float,1024,3000,300,10,10,6,5>, (const void*)&axis_pass_any<float,1024,false,3000,300,10,10,6,5>, nullptr, nullptr, 1024, 0},
  {3456, 288, 4, {12,6,6,8}, 1024, (const void*)&axis_pass_static<float,1024,3456,288,12,6,6,8>, (const void*)&axis_pass_any<float,1024,false,3456,288,12,6,6,8>, nullptr, nullptr, 1024, 0},
  {4000, 400, 4, {10,10,5,8}, 1024, (const void*)&axis_pass_static<float,1024,4000,400,10,10,5,8>, (const void*)&axis_pass_any<float,1024,false,4000,400,10,10,5,8>, nullptr, nullptr, 1024, 0},
};
const int kPlansCount_f32_5 = 49;
}  // namespace dfft
