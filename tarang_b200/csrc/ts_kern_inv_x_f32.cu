#define TS_REAL float
#define TS_PART TS_PART_IX
#include "ts_kern_impl.cuh"
