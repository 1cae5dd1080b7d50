// Kernels of the panda robot (generated FK and checks in robots/panda.cuh).
#include "robots/panda.cuh"
#include "vg_robot.cuh"

// same-edge schedule, built for the robot's own number of resident blocks
VG_DEFINE_ROBOT(Panda, ops_panda, 1)
