// Mixed precision, zero torque: every stepper and evaluation kernel.
#include "bd_tables.cuh"

bd::KernelTable bd::table_mixed() { return make_table<float, false>(); }
