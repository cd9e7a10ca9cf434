// The order in which a block's computing warps take key stages from the ring that lse_decode_layers' data comes through: where a
// stage lies, which warp works on it, and when each of them waits and gives it back.  Compiles for the host too.
#pragma once

#ifdef __CUDACC__
#define LSE_RING_FN __device__ __forceinline__
#else
#define LSE_RING_FN inline
#endif

// A place in the ring and the parity of its barriers' phase.
struct Slot {
  int at = 0;
  unsigned parity = 0;
  LSE_RING_FN void step(int stages) {
    if (++at == stages) { at = 0; parity ^= 1u; }
  }
};

// One warp's way through the stages of `tiles` tiles, `a_stage` of them a stage, `warps` (a power of two) warps taking the tiles in
// turn: work(slot, i, t) for tile t, the i-th of its stage.
// Every warp waits for every stage, also for those of which it has no tile: `done` counts its arrival for the phase that the
// stage's data opens.  A warp that did not wait could arrive for the slot's next use while another still reads this one; the
// early arrival would complete the count, and the slot would be filled again under that other warp.
template <typename Wait, typename Work, typename Done>
LSE_RING_FN void walk_key_stages(int warp, int warps, int tiles, int a_stage, int stages, Slot& slot, Wait wait, Work work, Done done) {
#ifdef __CUDACC__
#pragma unroll 1
#endif
  for (int first = 0; first < tiles; first += a_stage) {
    const int i = (warp - first) & (warps - 1), t = first + i;
    wait(slot);
    if (i < a_stage && t < tiles) work(slot, i, t);
    done(slot);
    slot.step(stages);
  }
}
