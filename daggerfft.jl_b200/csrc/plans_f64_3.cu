// Generated by gen_plans.py -- do not edit.
#include "static_plans.h"
namespace dfft {
template __global__ void axis_pass_static<double,1024,4,1,4>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,4,1,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,10,1,10>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,10,1,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,10,1,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,10,1,10>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,16,1,16>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,16,1,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,16,1,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,16,1,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,1024,25,5,5,5>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,25,5,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,25,5,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,25,5,5,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,33,3,11,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,33,3,11,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,44,4,11,4>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,44,4,11,4>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,54,9,6,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,54,9,6,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,54,9,6,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,54,9,6,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,65,5,13,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,65,5,13,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,78,6,13,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,78,6,13,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,91,7,13,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,91,7,13,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,105,7,15,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,105,7,15,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,121,11,11,11>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,121,11,11,11>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,135,9,15,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,135,9,15,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,135,9,15,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,135,9,15,3,3>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,154,11,14,11>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,154,11,14,11>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,169,13,13,13>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,169,13,13,13>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,192,12,12,16>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,192,12,12,16>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,192,12,12,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,192,12,12,16>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,256,210,14,15,14>(const PassDesc);
template __global__ void axis_pass_any<double,256,false,210,14,15,14>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,234,18,13,6,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,234,18,13,6,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,252,36,7,6,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,252,36,7,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,275,25,11,5,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,275,25,11,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,300,30,10,6,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,300,30,10,6,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,300,30,10,6,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,300,30,10,6,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,325,25,13,5,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,325,25,13,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,351,27,13,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,351,27,13,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,378,54,7,6,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,378,54,7,6,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,400,40,10,5,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,400,40,10,5,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,400,40,10,5,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,400,40,10,5,8>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,440,40,11,5,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,440,40,11,5,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,468,36,13,6,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,468,36,13,6,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,500,50,10,10,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,500,50,10,10,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_pipe<double,512,false,8,500,50,10,10,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_pipe<double,512,true,0,500,50,10,10,5>(const PassDesc, const __grid_constant__ CUtensorMap, const __grid_constant__ CUtensorMap, const TmaGeom);
template __global__ void axis_pass_static<double,512,528,48,11,6,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,528,48,11,6,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,567,81,7,3,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,567,81,7,3,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,600,60,10,10,6>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,600,60,10,10,6>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,637,49,13,7,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,637,49,13,7,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,675,45,15,15,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,675,45,15,15,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,704,64,11,8,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,704,64,11,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,735,49,15,7,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,735,49,15,7,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,784,56,14,7,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,784,56,14,7,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,832,64,13,8,8>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,832,64,13,8,8>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,875,125,7,5,5,5>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,875,125,7,5,5,5>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,910,70,13,10,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,910,70,13,10,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,1024,972,162,6,6,3,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,1024,false,972,162,6,6,3,3,3>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1008,84,12,12,7>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1008,84,12,12,7>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1200,100,12,10,10>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1200,100,12,10,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1440,120,12,12,10>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1440,120,12,12,10>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,1728,144,12,12,12>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,1728,144,12,12,12>(const __grid_constant__ PassDesc);
template __global__ void axis_pass_static<double,512,2025,135,15,15,3,3>(const PassDesc);
template __global__ void axis_pass_any<double,512,false,2025,135,15,15,3,3>(const __grid_constant__ PassDesc);
extern const StaticPlan kPlans_f64_3[];
extern const int kPlansCount_f64_3;
const StaticPlan kPlans_f64_3[] = {
  {4, 1, 1, {4}, 1024, (const void*)&axis_pass_static<double,1024,4,1,4>, (const void*)&axis_pass_any<double,1024,false,4,1,4>, nullptr, nullptr, 512, 0},
  {10, 1, 1, {10}, 512, (const void*)&axis_pass_static<double,512,10,1,10>, (const void*)&axis_pass_any<double,512,false,10,1,10>, (const void*)&axis_pass_pipe<double,512,false,8,10,1,10>, (const void*)&axis_pass_pipe<double,512,true,0,10,1,10>, 512, 8},
  {16, 1, 1, {16}, 512, (const void*)&axis_pass_static<double,512,16,1,16>, (const void*)&axis_pass_any<double,512,false,16,1,16>, (const void*)&axis_pass_pipe<double,512,false,8,16,1,16>, (const void*)&axis_pass_pipe<double,512,true,0,16,1,16>, 512, 8},
  {25, 5, 2, {5,5}, 1024, (const void*)&axis_pass_static<double,1024,25,5,5,5>, (const void*)&axis_pass_any<double,1024,false,25,5,5,5>, (const void*)&axis_pass_pipe<double,512,false,8,25,5,5,5>, (const void*)&axis_pass_pipe<double,512,true,0,25,5,5,5>, 512, 8},
  {33, 3, 2, {11,3}, 512, (const void*)&axis_pass_static<double,512,33,3,11,3>, (const void*)&axis_pass_any<double,512,false,33,3,11,3>, nullptr, nullptr, 512, 0},
  {44, 4, 2, {11,4}, 512, (const void*)&axis_pass_static<double,512,44,4,11,4>, (const void*)&axis_pass_any<double,512,false,44,4,11,4>, nullptr, nullptr, 512, 0},
  {54, 9, 3, {6,3,3}, 1024, (const void*)&axis_pass_static<double,1024,54,9,6,3,3>, (const void*)&axis_pass_any<double,1024,false,54,9,6,3,3>, (const void*)&axis_pass_pipe<double,512,false,8,54,9,6,3,3>, (const void*)&axis_pass_pipe<double,512,true,0,54,9,6,3,3>, 512, 8},
  {65, 5, 2, {13,5}, 512, (const void*)&axis_pass_static<double,512,65,5,13,5>, (const void*)&axis_pass_any<double,512,false,65,5,13,5>, nullptr, nullptr, 512, 0},
  {78, 6, 2, {13,6}, 512, (const void*)&axis_pass_static<double,512,78,6,13,6>, (const void*)&axis_pass_any<double,512,false,78,6,13,6>, nullptr, nullptr, 512, 0},
  {91, 7, 2, {13,7}, 512, (const void*)&axis_pass_static<double,512,91,7,13,7>, (const void*)&axis_pass_any<double,512,false,91,7,13,7>, nullptr, nullptr, 512, 0},
  {105, 7, 2, {15,7}, 512, (const void*)&axis_pass_static<double,512,105,7,15,7>, (const void*)&axis_pass_any<double,512,false,105,7,15,7>, nullptr, nullptr, 512, 0},
  {121, 11, 2, {11,11}, 512, (const void*)&axis_pass_static<double,512,121,11,11,11>, (const void*)&axis_pass_any<double,512,false,121,11,11,11>, nullptr, nullptr, 512, 0},
  {135, 9, 3, {15,3,3}, 512, (const void*)&axis_pass_static<double,512,135,9,15,3,3>, (const void*)&axis_pass_any<double,512,false,135,9,15,3,3>, (const void*)&axis_pass_pipe<double,512,false,8,135,9,15,3,3>, (const void*)&axis_pass_pipe<double,512,true,0,135,9,15,3,3>, 512, 8},
  {154, 11, 2, {14,11}, 512, (const void*)&axis_pass_static<double,512,154,11,14,11>, (const void*)&axis_pass_any<double,512,false,154,11,14,11>, nullptr, nullptr, 512, 0},
  {169, 13, 2, {13,13}, 512, (const void*)&axis_pass_static<double,512,169,13,13,13>, (const void*)&axis_pass_any<double,512,false,169,13,13,13>, nullptr, nullptr, 512, 0},
  {192, 12, 2, {12,16}, 512, (const void*)&axis_pass_static<double,512,192,12,12,16>, (const void*)&axis_pass_any<double,512,false,192,12,12,16>, (const void*)&axis_pass_pipe<double,512,false,8,192,12,12,16>, (const void*)&axis_pass_pipe<double,512,true,0,192,12,12,16>, 512, 8},
  {210, 14, 2, {15,14}, 256, (const void*)&axis_pass_static<double,256,210,14,15,14>, (const void*)&axis_pass_any<double,256,false,210,14,15,14>, nullptr, nullptr, 256, 0},
  {234, 18, 3, {13,6,3}, 512, (const void*)&axis_pass_static<double,512,234,18,13,6,3>, (const void*)&axis_pass_any<double,512,false,234,18,13,6,3>, nullptr, nullptr, 512, 0},
  {252, 36, 3, {7,6,6}, 512, (const void*)&axis_pass_static<double,512,252,36,7,6,6>, (const void*)&axis_pass_any<double,512,false,252,36,7,6,6>, nullptr, nullptr, 512, 0},
  {275, 25, 3, {11,5,5}, 512, (const void*)&axis_pass_static<double,512,275,25,11,5,5>, (const void*)&axis_pass_any<double,512,false,275,25,11,5,5>, nullptr, nullptr, 512, 0},
  {300, 30, 3, {10,6,5}, 512, (const void*)&axis_pass_static<double,512,300,30,10,6,5>, (const void*)&axis_pass_any<double,512,false,300,30,10,6,5>, (const void*)&axis_pass_pipe<double,512,false,8,300,30,10,6,5>, (const void*)&axis_pass_pipe<double,512,true,0,300,30,10,6,5>, 512, 8},
  {325, 25, 3, {13,5,5}, 512, (const void*)&axis_pass_static<double,512,325,25,13,5,5>, (const void*)&axis_pass_any<double,512,false,325,25,13,5,5>, nullptr, nullptr, 512, 0},
  {351, 27, 4, {13,3,3,3}, 512, (const void*)&axis_pass_static<double,512,351,27,13,3,3,3>, (const void*)&axis_pass_any<double,512,false,351,27,13,3,3,3>, nullptr, nullptr, 512, 0},
  {378, 54, 4, {7,6,3,3}, 512, (const void*)&axis_pass_static<double,512,378,54,7,6,3,3>, (const void*)&axis_pass_any<double,512,false,378,54,7,6,3,3>, nullptr, nullptr, 512, 0},
  {400, 40, 3, {10,5,8}, 512, (const void*)&axis_pass_static<double,512,400,40,10,5,8>, (const void*)&axis_pass_any<double,512,false,400,40,10,5,8>, (const void*)&axis_pass_pipe<double,512,false,8,400,40,10,5,8>, (const void*)&axis_pass_pipe<double,512,true,0,400,40,10,5,8>, 512, 8},
  {440, 40, 3, {11,5,8}, 512, (const void*)&axis_pass_static<double,512,440,40,11,5,8>, (const void*)&axis_pass_any<double,512,false,440,40,11,5,8>, nullptr, nullptr, 512, 0},
  {468, 36, 3, {13,6,6}, 512, (const void*)&axis_pass_static<double,512,468,36,13,6,6>, (const void*)&axis_pass_any<double,512,false,468,36,13,6,6>, nullptr, nullptr, 512, 0},
  {500, 50, 3, {10,10,5}, 512, (const void*)&axis_pass_static<double,512,500,50,10,10,5>, (const void*)&axis_pass_any<double,512,false,500,50,10,10,5>, (const void*)&axis_pass_pipe<double,512,false,8,500,50,10,10,5>, (const void*)&axis_pass_pipe<double,512,true,0,500,50,10,10,5>, 512, 8},
  {528, 48, 3, {11,6,8}, 512, (const void*)&axis_pass_static<double,512,528,48,11,6,8>, (const void*)&axis_pass_any<double,512,false,528,48,11,6,8>, nullptr, nullptr, 512, 0},
  {567, 81, 5, {7,3,3,3,3}, 512, (const void*)&axis_pass_static<double,512,567,81,7,3,3,3,3>, (const void*)&axis_pass_any<double,512,false,567,81,7,3,3,3,3>, nullptr, nullptr, 512, 0},
  {600, 60, 3, {10,10,6}, 512, (const void*)&axis_pass_static<double,512,600,60,10,10,6>, (const void*)&axis_pass_any<double,512,false,600,60,10,10,6>, nullptr, nullptr, 512, 0},
  {637, 49, 3, {13,7,7}, 512, (const void*)&axis_pass_static<double,512,637,49,13,7,7>, (const void*)&axis_pass_any<double,512,false,637,49,13,7,7>, nullptr, nullptr, 512, 0},
  {675, 45, 3, {15,15,3}, 512, (const void*)&axis_pass_static<double,512,675,45,15,15,3>, (const void*)&axis_pass_any<double,512,false,675,45,15,15,3>, nullptr, nullptr, 512, 0},
  {704, 64, 3, {11,8,8}, 512, (const void*)&axis_pass_static<double,512,704,64,11,8,8>, (const void*)&axis_pass_any<double,512,false,704,64,11,8,8>, nullptr, nullptr, 512, 0},
  {735, 49, 3, {15,7,7}, 512, (const void*)&axis_pass_static<double,512,735,49,15,7,7>, (const void*)&axis_pass_any<double,512,false,735,49,15,7,7>, nullptr, nullptr, 512, 0},
  {784, 56, 3, {14,7,8}, 512, (const void*)&axis_pass_static<double,512,784,56,14,7,8>, (const void*)&axis_pass_any<double,512,false,784,56,14,7,8>, nullptr, nullptr, 512, 0},
  {832, 64, 3, {13,8,8}, 512, (const void*)&axis_pass_static<double,512,832,64,13,8,8>, (const void*)&axis_pass_any<double,512,false,832,64,13,8,8>, nullptr, nullptr, 512, 0},
  {875, 125, 4, {7,5,5,5}, 512, (const void*)&axis_pass_static<double,512,875,125,7,5,5,5>, (const void*)&axis_pass_any<double,512,false,875,125,7,5,5,5>, nullptr, nullptr, 512, 0},
  {910, 70, 3, {13,10,7}, 512, (const void*)&axis_pass_static<double,512,910,70,13,10,7>, (const void*)&axis_pass_any<double,512,false,910,70,13,10,7>, nullptr, nullptr, 512, 0},
  {972, 162, 5, {6,6,3,3,3}, 1024, (const void*)&axis_pass_static<double,1024,972,162,6,6,3,3,3>, (const void*)&axis_pass_any<double,1024,false,972,162,6,6,3,3,3>, nullptr, nullptr, 512, 0},
  {1008, 84, 3, {12,12,7}, 512, (const void*)&axis_pass_static<double,512,1008,84,12,12,7>, (const void*)&axis_pass_any<double,512,false,1008,84,12,12,7>, nullptr, nullptr, 512, 0},
  {1200, 100, 3, {12,10,10}, 512, (const void*)&axis_pass_static<double,512,1200,100,12,10,10>, (const void*)&axis_pass_any<double,512,false,1200,100,12,10,10>, nullptr, nullptr, 512, 0},
  {1440, 120, 3, {12,12,10}, 512, (const void*)&axis_pass_static<double,512,1440,120,12,12,10>, (const void*)&axis_pass_any<double,512,false,1440,120,12,12,10>, nullptr, nullptr, 512, 0},
  {1728, 144, 3, {12,12,12}, 512, (const void*)&axis_pass_static<double,512,1728,144,12,12,12>, (const void*)&axis_pass_any<double,512,false,1728,144,12,12,12>, nullptr, nullptr, 512, 0},
  {2025, 135, 4, {15,15,3,3}, 512, (const void*)&axis_pass_static<double,512,2025,135,15,15,3,3>, (const void*)&axis_pass_any<double,512,false,2025,135,15,15,3,3>, nullptr, nullptr, 512, 0},
};
const int kPlansCount_f64_3 = 45;
}  // namespace dfft
