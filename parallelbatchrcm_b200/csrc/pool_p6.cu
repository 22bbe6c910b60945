// pool_p6.cu -- batch kernels of pool shape 6: 256-thread CTAs of one group with 1024-edge chunks; the solo batch
// kernel two per SM (128 registers).  What a third group adds in flight it takes from the others' share of L2 (the
// matrices' edge records and positions are read at random): 4,096 mixed matrices 66.4 ms with three CTAs of 80
// registers, 58.6 with two; 73.2 with one CTA of 512 threads.  Three per SM all the same where that saves equal
// matrices a round (run_batch): 444 27-point meshes of 7,200 nodes 3.25 ms with three, 4.98 with two.
#include "pool.cuh"

PBRCM_DEFINE_POOL_MORE(6, 256, 1024, 256, 1024, 3, 2, 3)
