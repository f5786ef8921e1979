// FP64, torque about the centroid: every stepper and evaluation kernel.
#include "bd_tables.cuh"

bd::KernelTable bd::table_fp64_torque() { return make_table<double, true>(); }
