#define TS_REAL double
#define TS_PART TS_PART_IX
#include "ts_kern_impl.cuh"
