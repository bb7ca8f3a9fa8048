#define TS_REAL float
#define TS_PART TS_PART_MISC
#include "ts_kern_impl.cuh"
