// coop_share.h — how many blocks a batch worker's cooperative launch may have.
//
// Workers run side by side, and a cooperative kernel's blocks wait for one
// another: a launch that finds places for some of its blocks only, because the
// others' blocks lie badly, waits half resident until another worker's kernel
// ends, and its wait budget runs.  The two cooperative kernels are the grouping
// (256 threads of 128 registers: half an SM) and the ICP of a worker (256 of 64:
// a quarter).  ICP blocks fit wherever registers are free; a grouping block
// wants half an SM, and j quarters on an SM leave it floor((4 - j) / 2) places:
// one ICP block costs as much as two.  The shares below fit for any number of
// workers in either kernel, wherever the blocks lie: k workers' ICPs hold at
// most 3 k S / n quarters of S SMs and so cost at most (3 k S / n + S) / 2 of the
// 2 S half places, which leaves the other n - k their 3 S / 2 n each.
// Where an SM's shared memory holds one grouping block only (correspondences in
// the hundreds of thousands), a block of either kind may spoil its SM for
// others: a worker gets S / n blocks.
// This counts registers and shared memory, as the occupancy calculation does;
// how the hardware orders blocks of several grids is its own, so waits keep
// their budget.
#pragma once

namespace rtr {

struct CoopShare {
  int icp, gc;
};

// sms: the GPU's; workers: that run side by side (at least 2); gc_per_sm:
// grouping blocks that an SM holds (2, or 1).
constexpr CoopShare coop_share(int sms, int workers, int gc_per_sm) {
  return gc_per_sm >= 2 ? CoopShare{3 * sms / workers, 3 * sms / (2 * workers)}
                        : CoopShare{sms / workers, sms / workers};
}

}  // namespace rtr
