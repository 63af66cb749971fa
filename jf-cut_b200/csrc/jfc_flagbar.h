// jfc_flagbar.h — the word of a grid barrier that also tells every block whether
// any block asked for a next phase.  Plain functions, host and device: the CPU
// tests run the protocol through every order of arrivals and polls.
#pragma once

#ifdef __CUDACC__
#define JFC_HD __host__ __device__
#else
#define JFC_HD
#endif

namespace jfc {

// The word: arrivals since the launch began (bits 0-39, they only grow), and
// two counts of 12 bits, the blocks whose last arrival at an even (bits 40-51) /
// odd (52-63) barrier asked for a next phase.  A block replaces its own share
// of a count when it arrives at the next barrier of that parity.  No block
// is more than one barrier ahead of the slowest, so while a block still polls
// for barrier b the others can only have changed the other parity's count: it
// reads barrier b's, however late its poll.  (One count that grew over all
// barriers, compared with what the block last saw, mixed the two: a late poller
// took the next barrier's requests for this one's, missed them at the next,
// and left alone.)
constexpr unsigned kFlagBarBlocks = 4095;   // most blocks of a launch

struct FlagBar {
  // What a block adds to arrive at barrier b (0, 1, 2, ...).  mine: the parities at
  // which its last arrival asked, 0 at the launch's start.
  static JFC_HD unsigned long long arrival(unsigned b, bool ask, unsigned& mine) {
    const unsigned was = mine >> (b & 1u) & 1u;
    mine ^= (was ^ (ask ? 1u : 0u)) << (b & 1u);
    return 1ull + (((ask ? 1ull : 0ull) - was) << shift(b));
  }
  // Barrier b is complete: all of its arrivals of `blocks` blocks are in.
  static JFC_HD bool complete(unsigned long long word, unsigned b, unsigned blocks) {
    return (word & ((1ull << 40) - 1)) >= ((unsigned long long)b + 1) * blocks;
  }
  // Some block asked at barrier b (complete, and the caller not arrived at b + 1).
  static JFC_HD bool asked(unsigned long long word, unsigned b) { return (word >> shift(b) & 0xfffu) != 0; }

 private:
  static JFC_HD unsigned shift(unsigned b) { return b & 1u ? 52u : 40u; }
};

}  // namespace jfc
