// What csrc/api.cu and its headers need from nvcc, for a host compiler: names of
// device functions that no host code calls, and min and max.
#pragma once
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <algorithm>
#include <cstdint>
#include <cstdlib>
using std::max;
using std::min;
int __double2loint(double);
int __double2hiint(double);
double __dmul_rn(double, double);
double __ddiv_rn(double, double);
double __fma_rn(double, double, double);
template <class T>
T __ldg(const T*);
void fake_launch(cudaStream_t st);  // in place of a kernel launch
