// The steps that the multiplying warps of the packed-expert product (moe_fp4.cu) take together through one pass. Plain C++: the kernel
// compiles it for the device, a test for threads of the host.
#pragma once

#ifdef __CUDACC__
#define FF_WALK __device__ __forceinline__
#else
#define FF_WALK inline
#endif

namespace ff {

// chunks: ring stages of the pass; per_slab: stages that the tokens in shared memory cover. meet(): barrier of all warps; fill(c): tokens of
// the slab that begins with chunk c; wait(c): the stage has come (false: the wait gave up); multiply(c); meet_any(f): barrier that tells
// every warp whether any passed true. Returns whether the pass holds, the same to all warps.
// A barrier counts all warps and has no limit of its own. So a warp whose wait gave up stays in step: it fills and multiplies nothing more,
// meets the others at every barrier of the pass, and all of them leave together at the last one. (With that path inside the loop a product
// of 128 experts of 4096 x 1536 with two rows each took 136.3 us, with it apart 132.4.)
template <class Meet, class Fill, class Wait, class Multiply, class MeetAny>
FF_WALK bool walk_pass(int chunks, int per_slab, Meet meet, Fill fill, Wait wait, Multiply multiply, MeetAny meet_any) {
  for (int c = 0; c < chunks; ++c) {
    if (c % per_slab == 0) {
      meet();
      fill(c);
      meet();
    }
    if (!wait(c)) {
      for (++c; c < chunks; ++c)
        if (c % per_slab == 0) {
          meet();
          meet();
        }
      meet_any(true);
      return false;
    }
    multiply(c);
  }
  return !meet_any(false);
}

}  // namespace ff
