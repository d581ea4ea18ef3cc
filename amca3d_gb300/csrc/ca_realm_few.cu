// ca_realm_few.cu — the persistent plain kernel for realms run with at most one
// block per SM (ca_plain.cu compiled once more; see plain_run_steps).
#define AMCA_BLOCK 256
#define AMCA_MIN_BLOCKS 2
#define AMCA_REALM_FEW
#include "ca_plain.cu"
