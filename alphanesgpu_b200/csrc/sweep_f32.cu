#define REAL float
#include "sweep_launch.cuh"
