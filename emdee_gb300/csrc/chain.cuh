// chain.cuh -- launches that overlap the end of the kernel before them.
//
// A time step of a small system is a chain of short dependent kernels, and each boundary
// of an ordinary launch costs the drain of one grid and the start of the next.  launch_chained
// lets a grid start when every block of the grid before it has passed chain_wait; its
// own chain_wait, the first statement of the kernel, holds it until that grid has
// completed and its writes are visible.  Per pass of 10 to 20 steps: 800 atoms 787 -> 703 us,
// 512 flexible waters 712 -> 650, 4096 rigid waters 862 -> 793, 16,001 atoms 623 -> 601,
// 1,048,576 atoms 3390 -> 3305.  Not on a side stream: blocks that wait there hold places
// that the pair kernel on the main stream needs (1000 waters with Ewald sums 1074 -> 1114
// us with its sums chained, 1033 without).  Kernels launched the ordinary way are ordered as
// always, whatever is before or behind them, and chain_wait returns at once in them.
//
// A kernel that is launched so starts while the one before it still writes.  What any kernel
// writes is therefore not declared `const T* __restrict__` there, nor read by __ldg: both
// promise memory that nobody writes while the kernel runs, and such a load may be moved
// in front of the wait or served from a line read before it.  Only arrays that the host set up
// (masses, charges, species) are.
#pragma once
#include <utility>

#include "system.hpp"

namespace emdee {

// Blocks of a grid that let the next one start early.  The trigger goes through one counter
// at about two blocks per ns, which short blocks of a large grid wait for (244,000 blocks
// that return at once: 127 us without it, 252 with it; 61,000 blocks of the cell sort 41 and
// 65 us), and the overlap gains 2 to 3 us: above this line the next grid starts when this one
// has completed.
constexpr unsigned int CHAIN_BLOCKS = 8192;

__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (gridDim.x <= CHAIN_BLOCKS) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Whether a grid of this many long blocks (the list build, the pair kernels) is launched
// chained.  Its blocks take their places while the grid before them still holds some, so with
// one to a few blocks per SM the SMs that were free first end up with two while others have
// none.  In the steps themselves the overlap outweighs that: at a fixed tile edge, 10 steps
// are 4 to 6 % faster chained at 216 and 343 tiles, 3 to 4 % at 512 and 729, 2 to 3 % at 1000 to
// 1728, 7 to 10 % at 27 to 125.  But the tuner times launches one at a time behind a pass over memory,
// where it sees only the uneven placement (50,021 atoms of two types on 180 tiles of 3 cells:
// 54 us chained, 50.5 not, 50 on the few tiles of 5 cells), and would leave the edge that is better
// in the steps (800 us for 10) for the other (880).  So grids between one block per SM
// and four are launched the ordinary way.
inline bool chain_fits(int blocks) { return blocks <= 152 || blocks >= 4 * 152; }

template <class... P, class... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... a) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  c.attrs = attr;
  c.numAttrs = 1;
  CK(cudaLaunchKernelEx(&c, kernel, P(std::forward<A>(a))...));
}

}  // namespace emdee
