// How one request's keys are cut in a decode attention launch (attention_mma.cu).
#pragma once

// The launch gives every (request, kv head) `launch_blocks` blocks of `warps` warps, cut for the step's longest request:
// `launch_keys` keys a warp, in tiles of `tile`.  A request spreads its `span` keys evenly over the warps of its blocks, at least 64
// a warp (or the launch's cut, if that is shorter); with the launch's cut for all, a request of a quarter of the longest one's
// keys leaves three warps in four of its block idle (64 requests of 250 to 1,750 keys, heads of 64: 48.8 us a layer, 44.0 so).
// How many blocks it takes depends on whether the whole launch has places at once, two blocks an SM (`spread`).  If so, all of
// them: nobody waits for the places, and the shorter its part, the sooner a warp is done (4 requests of 2,048 keys, window 512,
// heads of 128: 10.8 us over all blocks, 13.2 over as many as the launch's cut would fill).  If not, as many as the launch's
// cut would fill: the others leave at once and make room (21 requests of 512 to 3,500 keys, heads of 64, two blocks each:
// 33.3 us over all blocks, 24.9 so; with the launch's cut inside the blocks as well 26.3).
#ifdef __CUDACC__
#define IE_SPLIT_FN __host__ __device__ __forceinline__
#else
#define IE_SPLIT_FN static inline
#endif
// Keys of a warp, whole tiles.
IE_SPLIT_FN int decode_split_keys(int span, int launch_keys, int launch_blocks, bool spread, const int warps, const int tile) {
  const int least = launch_keys < 64 ? launch_keys : 64;
  int blocks = launch_blocks;
  if (launch_blocks > 1 && !spread) {
    blocks = (span + launch_keys * warps - 1) / (launch_keys * warps);
    blocks = blocks < 1 ? 1 : (blocks > launch_blocks ? launch_blocks : blocks);
  }
  const int even = blocks == 1 ? (span + warps - 1) / warps : (span + blocks * warps - 1) / (blocks * warps);
  const int whole = (even + tile - 1) / tile * tile;
  return whole > least ? whole : least;
}

// Blocks that hold some of the request's keys: the first ones (a block's own answer, block * warps * keys < span, needs no division).
IE_SPLIT_FN int decode_split_blocks(int span, int keys, const int warps) {
  return span <= keys * warps ? 1 : (span + keys * warps - 1) / (keys * warps);
}
