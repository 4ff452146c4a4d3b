#define REAL double
#include "mlp_launch.cuh"
