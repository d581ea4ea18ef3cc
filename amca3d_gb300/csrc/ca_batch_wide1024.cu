// ca_batch_wide1024.cu — the batched plain kernel with blocks of 1024 threads
// (ca_plain.cu compiled once more; see plain_batched_threads).
#define AMCA_BLOCK 1024
#define AMCA_MIN_BLOCKS 1
#define AMCA_BATCH_WIDE plain_batched_launch_1024
#define AMCA_BATCH_WIDE_GRID plain_batched_grid_1024
#include "ca_plain.cu"
