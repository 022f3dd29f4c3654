// Which K blocks an MMA-issuing thread takes, and where they lie in the ring. Plain C++, shared by the kernel and a host test.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define ISSUER_WALK_FN __host__ __device__ __forceinline__
#else
#define ISSUER_WALK_FN inline
#endif

// "Block" here is one use of the ring: a K block, or the two that share a stage at 64-wide tiles, where both MMA threads walk every
// use (issuers = 1) and take a K block of it each.
// Block j of a CTA's whole sequence lies in ring stage j mod stages and TMEM buffer j mod buffers. Issuer `me` of `issuers`
// takes the blocks of stages me, me + issuers, ...: every issuers-th block while the number of stages is a multiple of
// `issuers`, and at the end of an odd ring of two the next block follows at once.
//
// A stage has ONE issuer because a barrier wait tells only the parity of a phase: a thread that waits for use n of a stage
// must have seen use n - 1 complete, or it takes "use n - 1 is still outstanding" for "use n is complete". With every second
// block to each issuer, the stages of an odd ring change hands, and an issuer whose own blocks had landed first issued MMAs on
// a stage whose copies were still in flight (128-wide tiles then ran five stages).
struct IssuerWalk {
  int stage, buffer;
  uint32_t phase;
  int block;  // offset of the next K block from the start of the current tile

  ISSUER_WALK_FN void begin(int me, int stages, int buffers) {
    stage = me;
    buffer = me % buffers;
    phase = 0;
    block = me;
    (void)stages;
  }
  ISSUER_WALK_FN void next(int me, int issuers, int stages, int buffers) {
    int step = issuers;
    stage += issuers;
    if (stage >= stages) {
      step = stages - stage + issuers + me;  // from the last stage of this issuer to its first one in the next round
      stage = me;
      phase ^= 1u;
    }
    block += step;
    buffer += step;
    while (buffer >= buffers) buffer -= buffers;
  }
};
