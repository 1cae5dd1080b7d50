// Kernels of the baxter robot (generated FK and checks in robots/baxter.cuh).
#include "robots/baxter.cuh"
#include "vg_robot.cuh"

// same-edge schedule, built for the robot's own number of resident blocks
VG_DEFINE_ROBOT(Baxter, ops_baxter, 1)
