#define TS_REAL double
#define TS_PART TS_PART_FX
#include "ts_kern_impl.cuh"
