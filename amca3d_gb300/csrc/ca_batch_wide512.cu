// ca_batch_wide512.cu — the batched plain kernel with blocks of 512 threads
// (ca_plain.cu compiled once more; see plain_batched_threads).
#define AMCA_BLOCK 512
#define AMCA_MIN_BLOCKS 2
#define AMCA_BATCH_WIDE plain_batched_launch_512
#define AMCA_BATCH_WIDE_GRID plain_batched_grid_512
#include "ca_plain.cu"
