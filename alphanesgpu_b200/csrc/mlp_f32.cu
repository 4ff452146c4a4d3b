#define REAL float
#include "mlp_launch.cuh"
