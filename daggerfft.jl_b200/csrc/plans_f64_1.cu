// Generated by gen_plans.py -- do not edit.
#include "static_plans.h"
namespace dfft {
template __global__ void axis_pass_static<double,1024,2,1,2>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,2,1,2>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,8,1,8>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,8,1,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,8,1,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,8,1,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,14,1,14>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,14,1,14>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,22,2,11,2>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,22,2,11,2>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,30,5,6,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,30,5,6,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,30,5,6,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,30,5,6,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,40,5,5,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,40,5,5,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,40,5,5,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,40,5,5,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,50,5,10,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,50,5,10,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,50,5,10,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,50,5,10,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,63,9,7,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,63,9,7,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,75,5,15,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,75,5,15,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,75,5,15,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,75,5,15,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,88,8,11,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,88,8,11,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,100,10,10,10>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,100,10,10,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,100,10,10,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,100,10,10,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,117,9,13,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,117,9,13,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,130,10,13,10>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,130,10,13,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,147,21,7,7,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,147,21,7,7,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,165,11,15,11>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,165,11,15,11>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,256,182,13,14,13>(const PassDesc);
template __global__ void axis_pass_any<double,256,false,182,13,14,13>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,200,25,5,5,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,200,25,5,5,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,200,25,5,5,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,200,25,5,5,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,225,15,15,15>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,225,15,15,15>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,225,15,15,15>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,225,15,15,15>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,245,35,7,7,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,245,35,7,7,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,270,18,15,6,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,270,18,15,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,270,18,15,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,270,18,15,6,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,294,42,7,7,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,294,42,7,7,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,320,40,5,8,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,320,40,5,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,320,40,5,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,320,40,5,8,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,1024,343,49,7,7,7>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,343,49,7,7,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,364,28,13,7,4>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,364,28,13,7,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,392,49,7,7,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,392,49,7,7,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,429,33,13,11,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,429,33,13,11,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,455,35,13,7,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,455,35,13,7,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,490,49,10,7,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,490,49,10,7,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,520,40,13,5,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,520,40,13,5,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,550,50,11,10,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,550,50,11,10,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,588,49,12,7,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,588,49,12,7,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,625,125,5,5,5,5>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,625,125,5,5,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,660,60,11,10,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,660,60,11,10,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,700,70,10,10,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,700,70,10,10,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,728,56,13,7,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,728,56,13,7,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,770,70,11,10,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,770,70,11,10,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,819,63,13,7,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,819,63,13,7,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,858,66,13,11,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,858,66,13,11,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,896,64,14,8,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,896,64,14,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,960,80,12,10,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,960,80,12,10,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1000,100,10,10,10>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1000,100,10,10,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1125,75,15,15,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1125,75,15,15,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,1296,216,6,6,6,6>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,1296,216,6,6,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1600,100,10,10,16>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1600,100,10,10,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,1944,324,6,6,6,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,1944,324,6,6,6,3,3>(const __grid_constant__ PassDesc);
extern const StaticPlan kPlans_f64_1[];
extern const int kPlansCount_f64_1;
const StaticPlan kPlans_f64_1[] = {
  {2, 1, 1, {2}, 1024, (const void*)&axis_pass_static<double,1024,2,1,2>, (const void*)&axis_pass_any<double,1024,false,2,1,2>, nullptr, nullptr, 512, 0},
  {8, 1, 1, {8}, 1024, (const void*)&axis_pass_static<double,1024,8,1,8>, (const void*)&axis_pass_any<double,1024,false,8,1,8>, (const void*)&axis_pass_pipe<double,512,false,8,8,1,8>, (const void*)&axis_pass_pipe<double,512,true,0,8,1,8>, 512, 8},
  {14, 1, 1, {14}, 512, (const void*)&axis_pass_static<double,512,14,1,14>, (const void*)&axis_pass_any<double,512,false,14,1,14>, nullptr, nullptr, 512, 0},
  {22, 2, 2, {11,2}, 512, (const void*)&axis_pass_static<double,512,22,2,11,2>, (const void*)&axis_pass_any<double,512,false,22,2,11,2>, nullptr, nullptr, 512, 0},
  {30, 5, 2, {6,5}, 512, (const void*)&axis_pass_static<double,512,30,5,6,5>, (const void*)&axis_pass_any<double,512,false,30,5,6,5>, (const void*)&axis_pass_pipe<double,512,false,8,30,5,6,5>, (const void*)&axis_pass_pipe<double,512,true,0,30,5,6,5>, 512, 8},
  {40, 5, 2, {5,8}, 512, (const void*)&axis_pass_static<double,512,40,5,5,8>, (const void*)&axis_pass_any<double,512,false,40,5,5,8>, (const void*)&axis_pass_pipe<double,512,false,8,40,5,5,8>, (const void*)&axis_pass_pipe<double,512,true,0,40,5,5,8>, 512, 8},
  {50, 5, 2, {10,5}, 512, (const void*)&axis_pass_static<double,512,50,5,10,5>, (const void*)&axis_pass_any<double,512,false,50,5,10,5>, (const void*)&axis_pass_pipe<double,512,false,8,50,5,10,5>, (const void*)&axis_pass_pipe<double,512,true,0,50,5,10,5>, 512, 8},
  {63, 9, 3, {7,3,3}, 512, (const void*)&axis_pass_static<double,512,63,9,7,3,3>, (const void*)&axis_pass_any<double,512,false,63,9,7,3,3>, nullptr, nullptr, 512, 0},
  {75, 5, 2, {15,5}, 512, (const void*)&axis_pass_static<double,512,75,5,15,5>, (const void*)&axis_pass_any<double,512,false,75,5,15,5>, (const void*)&axis_pass_pipe<double,512,false,8,75,5,15,5>, (const void*)&axis_pass_pipe<double,512,true,0,75,5,15,5>, 512, 8},
  {88, 8, 2, {11,8}, 512, (const void*)&axis_pass_static<double,512,88,8,11,8>, (const void*)&axis_pass_any<double,512,false,88,8,11,8>, nullptr, nullptr, 512, 0},
  {100, 10, 2, {10,10}, 512, (const void*)&axis_pass_static<double,512,100,10,10,10>, (const void*)&axis_pass_any<double,512,false,100,10,10,10>, (const void*)&axis_pass_pipe<double,512,false,8,100,10,10,10>, (const void*)&axis_pass_pipe<double,512,true,0,100,10,10,10>, 512, 8},
  {117, 9, 3, {13,3,3}, 512, (const void*)&axis_pass_static<double,512,117,9,13,3,3>, (const void*)&axis_pass_any<double,512,false,117,9,13,3,3>, nullptr, nullptr, 512, 0},
  {130, 10, 2, {13,10}, 512, (const void*)&axis_pass_static<double,512,130,10,13,10>, (const void*)&axis_pass_any<double,512,false,130,10,13,10>, nullptr, nullptr, 512, 0},
  {147, 21, 3, {7,7,3}, 512, (const void*)&axis_pass_static<double,512,147,21,7,7,3>, (const void*)&axis_pass_any<double,512,false,147,21,7,7,3>, nullptr, nullptr, 512, 0},
  {165, 11, 2, {15,11}, 512, (const void*)&axis_pass_static<double,512,165,11,15,11>, (const void*)&axis_pass_any<double,512,false,165,11,15,11>, nullptr, nullptr, 512, 0},
  {182, 13, 2, {14,13}, 256, (const void*)&axis_pass_static<double,256,182,13,14,13>, (const void*)&axis_pass_any<double,256,false,182,13,14,13>, nullptr, nullptr, 256, 0},
  {200, 25, 3, {5,5,8}, 512, (const void*)&axis_pass_static<double,512,200,25,5,5,8>, (const void*)&axis_pass_any<double,512,false,200,25,5,5,8>, (const void*)&axis_pass_pipe<double,512,false,8,200,25,5,5,8>, (const void*)&axis_pass_pipe<double,512,true,0,200,25,5,5,8>, 512, 8},
  {225, 15, 2, {15,15}, 512, (const void*)&axis_pass_static<double,512,225,15,15,15>, (const void*)&axis_pass_any<double,512,false,225,15,15,15>, (const void*)&axis_pass_pipe<double,512,false,8,225,15,15,15>, (const void*)&axis_pass_pipe<double,512,true,0,225,15,15,15>, 512, 8},
  {245, 35, 3, {7,7,5}, 512, (const void*)&axis_pass_static<double,512,245,35,7,7,5>, (const void*)&axis_pass_any<double,512,false,245,35,7,7,5>, nullptr, nullptr, 512, 0},
  {270, 18, 3, {15,6,3}, 512, (const void*)&axis_pass_static<double,512,270,18,15,6,3>, (const void*)&axis_pass_any<double,512,false,270,18,15,6,3>, (const void*)&axis_pass_pipe<double,512,false,8,270,18,15,6,3>, (const void*)&axis_pass_pipe<double,512,true,0,270,18,15,6,3>, 512, 8},
  {294, 42, 3, {7,7,6}, 512, (const void*)&axis_pass_static<double,512,294,42,7,7,6>, (const void*)&axis_pass_any<double,512,false,294,42,7,7,6>, nullptr, nullptr, 512, 0},
  {320, 40, 3, {5,8,8}, 512, (const void*)&axis_pass_static<double,512,320,40,5,8,8>, (const void*)&axis_pass_any<double,512,false,320,40,5,8,8>, (const void*)&axis_pass_pipe<double,512,false,8,320,40,5,8,8>, (const void*)&axis_pass_pipe<double,512,true,0,320,40,5,8,8>, 512, 8},
  {343, 49, 3, {7,7,7}, 1024, (const void*)&axis_pass_static<double,1024,343,49,7,7,7>, (const void*)&axis_pass_any<double,1024,false,343,49,7,7,7>, nullptr, nullptr, 512, 0},
  {364, 28, 3, {13,7,4}, 512, (const void*)&axis_pass_static<double,512,364,28,13,7,4>, (const void*)&axis_pass_any<double,512,false,364,28,13,7,4>, nullptr, nullptr, 512, 0},
  {392, 49, 3, {7,7,8}, 512, (const void*)&axis_pass_static<double,512,392,49,7,7,8>, (const void*)&axis_pass_any<double,512,false,392,49,7,7,8>, nullptr, nullptr, 512, 0},
  {429, 33, 3, {13,11,3}, 512, (const void*)&axis_pass_static<double,512,429,33,13,11,3>, (const void*)&axis_pass_any<double,512,false,429,33,13,11,3>, nullptr, nullptr, 512, 0},
  {455, 35, 3, {13,7,5}, 512, (const void*)&axis_pass_static<double,512,455,35,13,7,5>, (const void*)&axis_pass_any<double,512,false,455,35,13,7,5>, nullptr, nullptr, 512, 0},
  {490, 49, 3, {10,7,7}, 512, (const void*)&axis_pass_static<double,512,490,49,10,7,7>, (const void*)&axis_pass_any<double,512,false,490,49,10,7,7>, nullptr, nullptr, 512, 0},
  {520, 40, 3, {13,5,8}, 512, (const void*)&axis_pass_static<double,512,520,40,13,5,8>, (const void*)&axis_pass_any<double,512,false,520,40,13,5,8>, nullptr, nullptr, 512, 0},
  {550, 50, 3, {11,10,5}, 512, (const void*)&axis_pass_static<double,512,550,50,11,10,5>, (const void*)&axis_pass_any<double,512,false,550,50,11,10,5>, nullptr, nullptr, 512, 0},
  {588, 49, 3, {12,7,7}, 512, (const void*)&axis_pass_static<double,512,588,49,12,7,7>, (const void*)&axis_pass_any<double,512,false,588,49,12,7,7>, nullptr, nullptr, 512, 0},
  {625, 125, 4, {5,5,5,5}, 1024, (const void*)&axis_pass_static<double,1024,625,125,5,5,5,5>, (const void*)&axis_pass_any<double,1024,false,625,125,5,5,5,5>, nullptr, nullptr, 512, 0},
  {660, 60, 3, {11,10,6}, 512, (const void*)&axis_pass_static<double,512,660,60,11,10,6>, (const void*)&axis_pass_any<double,512,false,660,60,11,10,6>, nullptr, nullptr, 512, 0},
  {700, 70, 3, {10,10,7}, 512, (const void*)&axis_pass_static<double,512,700,70,10,10,7>, (const void*)&axis_pass_any<double,512,false,700,70,10,10,7>, nullptr, nullptr, 512, 0},
  {728, 56, 3, {13,7,8}, 512, (const void*)&axis_pass_static<double,512,728,56,13,7,8>, (const void*)&axis_pass_any<double,512,false,728,56,13,7,8>, nullptr, nullptr, 512, 0},
  {770, 70, 3, {11,10,7}, 512, (const void*)&axis_pass_static<double,512,770,70,11,10,7>, (const void*)&axis_pass_any<double,512,false,770,70,11,10,7>, nullptr, nullptr, 512, 0},
  {819, 63, 4, {13,7,3,3}, 512, (const void*)&axis_pass_static<double,512,819,63,13,7,3,3>, (const void*)&axis_pass_any<double,512,false,819,63,13,7,3,3>, nullptr, nullptr, 512, 0},
  {858, 66, 3, {13,11,6}, 512, (const void*)&axis_pass_static<double,512,858,66,13,11,6>, (const void*)&axis_pass_any<double,512,false,858,66,13,11,6>, nullptr, nullptr, 512, 0},
  {896, 64, 3, {14,8,8}, 512, (const void*)&axis_pass_static<double,512,896,64,14,8,8>, (const void*)&axis_pass_any<double,512,false,896,64,14,8,8>, nullptr, nullptr, 512, 0},
  {960, 80, 3, {12,10,8}, 512, (const void*)&axis_pass_static<double,512,960,80,12,10,8>, (const void*)&axis_pass_any<double,512,false,960,80,12,10,8>, nullptr, nullptr, 512, 0},
  {1000, 100, 3, {10,10,10}, 512, (const void*)&axis_pass_static<double,512,1000,100,10,10,10>, (const void*)&axis_pass_any<double,512,false,1000,100,10,10,10>, nullptr, nullptr, 512, 0},
  {1125, 75, 3, {15,15,5}, 512, (const void*)&axis_pass_static<double,512,1125,75,15,15,5>, (const void*)&axis_pass_any<double,512,false,1125,75,15,15,5>, nullptr, nullptr, 512, 0},
  {1296, 216, 4, {6,6,6,6}, 1024, (const void*)&axis_pass_static<double,1024,1296,216,6,6,6,6>, (const void*)&axis_pass_any<double,1024,false,1296,216,6,6,6,6>, nullptr, nullptr, 512, 0},
  {1600, 100, 3, {10,10,16}, 512, (const void*)&axis_pass_static<double,512,1600,100,10,10,16>, (const void*)&axis_pass_any<double,512,false,1600,100,10,10,16>, nullptr, nullptr, 512, 0},
  {1944, 324, 5, {6,6,6,3,3}, 1024, (const void*)&axis_pass_static<double,1024,1944,324,6,6,6,3,3>, (const void*)&axis_pass_any<double,1024,false,1944,324,6,6,6,3,3>, nullptr, nullptr, 512, 0},
};
const int kPlansCount_f64_1 = 45;
}  // namespace dfft
