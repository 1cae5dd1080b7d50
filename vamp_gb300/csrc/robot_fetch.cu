// Kernels of the fetch robot (generated FK and checks in robots/fetch.cuh).
#include "robots/fetch.cuh"
#include "vg_robot.cuh"

// same-edge schedule, built for the robot's own number of resident blocks
VG_DEFINE_ROBOT(Fetch, ops_fetch, 1)
