#define REAL double
#include "sweep_launch.cuh"
