// Kernels of the ur5 robot (generated FK and checks in robots/ur5.cuh).
#include "robots/ur5.cuh"
#include "vg_robot.cuh"

// same-edge schedule, built for the robot's own number of resident blocks
VG_DEFINE_ROBOT(Ur5, ops_ur5, 1)
