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

// The last copy into `slot`, -1 if there was none: copies 0 .. n-1 were issued,
// and of the group of copies n, n+1, ... that was under way, those whose bits
// are set in `some` (the group holds fewer copies than there are slots).
XBG_RING_HD int ring_last(int n, unsigned some, int slots, int slot) {
    int c = slot - n % slots;   // the group's copy into this slot
    if (c < 0) c += slots;
    if (c < 32 && (some >> c & 1u)) return n + c;
    return n + c - slots < 0 ? -1 : n + c - slots;
}
// ... and the parity of the phase that it completes
XBG_RING_HD unsigned ring_parity(int copy, int slots) { return (unsigned)(copy / slots) & 1u; }

}  // namespace nn
}  // namespace xbg
