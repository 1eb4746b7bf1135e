// C entries of the copy ring's bookkeeping (csrc/copy_ring.cuh) for the test.
#include "copy_ring.cuh"
extern "C" int ring_last(int n, int slots, int slot) { return xbg::nn::ring_last(n, slots, slot); }
extern "C" unsigned ring_parity(int copy, int slots) { return xbg::nn::ring_parity(copy, slots); }
