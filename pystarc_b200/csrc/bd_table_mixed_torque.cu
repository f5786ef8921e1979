// Mixed precision, torque about the centroid: every stepper and evaluation kernel.
#include "bd_tables.cuh"

bd::KernelTable bd::table_mixed_torque() { return make_table<float, true>(); }
