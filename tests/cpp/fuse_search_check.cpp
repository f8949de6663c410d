// fuse_check.cpp with each block's qubits chosen by the search (same input and output).
#include "../../quaru_gb300/csrc/qs_fuse.h"

#define fuse_blocks(gates, m, W) fuse_blocks(gates, m, W, true)
#include "fuse_check.cpp"
