#define TS_REAL double
#define TS_PART TS_PART_MISC
#include "ts_kern_impl.cuh"
