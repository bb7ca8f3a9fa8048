#define TS_REAL float
#define TS_PART TS_PART_STR
#include "ts_kern_impl.cuh"
