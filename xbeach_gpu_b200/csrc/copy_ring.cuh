// The slots of a copy warp's ring.  Copies are numbered 0, 1, 2, ... in issue
// order; copy q goes to slot q % slots and completes phase q / slots of the
// slot's barrier.  A kernel that leaves early has to wait for the last copy into
// every slot: bulk copies complete in any order, so an older copy may land after
// a younger one, and a slot's last copy is the only one of the slot that may
// still be under way (the one before was waited for before the slot was reused).
#pragma once

#ifdef __CUDACC__
#define XBG_RING_HD __host__ __device__ inline
#else
#define XBG_RING_HD inline
#endif

namespace xbg {
namespace nn {

// The last of the copies 0 .. n-1 into `slot`, -1 if there was none.
XBG_RING_HD int ring_last(int n, int slots, int slot) {
    int c = slot - n % slots;   // copy n + c is the slot's next one
    if (c < 0) c += slots;
    return n + c - slots < 0 ? -1 : n + c - slots;
}
// ... and the parity of the phase that it completes
XBG_RING_HD unsigned ring_parity(int copy, int slots) { return (unsigned)(copy / slots) & 1u; }

}  // namespace nn
}  // namespace xbg
