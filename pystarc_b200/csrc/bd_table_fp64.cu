// FP64, zero torque: every stepper and evaluation kernel.
#include "bd_tables.cuh"

bd::KernelTable bd::table_fp64() { return make_table<double, false>(); }
