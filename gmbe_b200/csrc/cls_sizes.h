// Sizes of the bitmap tier's lists, levels and scratch, in 32-bit words: plain
// arithmetic, shared by the kernel, the scratch layout and the CPU tests.
#pragma once

#ifdef __CUDACC__
#define GMBE_HD __host__ __device__ __forceinline__
#else
#define GMBE_HD inline
#endif

namespace gmbe {

constexpr int kKMax = 4;         // bitmap words of a sub-problem
constexpr int kFrameWords = 32;  // a level's frame (ClsFrame)

GMBE_HD long long cls_stride(long long n) { return (n + 31) & ~31LL; }
// Words of a list of n classes with K-word masks (a multiple of 32).
GMBE_HD long long cls_list_words(long long n, int K) { return cls_stride(n) * (K + 3); }
// Words of a bit per class (an even number: what follows is 8-byte aligned).
GMBE_HD long long cls_bit_words(long long n) { return 2 * ((n + 63) >> 6); }
// A level: its frame, its L words and the live bits of its list's classes.
GMBE_HD long long cls_frame_words(long long n, int K) {
  return kFrameWords + cls_bit_words(n) + ((K + 1) & ~1);
}
// Most levels of a sub-problem: a level's L and its classes to push are both
// fewer than those of the level above.
GMBE_HD int cls_levels(int kn, int np) { return kn < np + 1 ? kn : np + 1; }
// Words a sub-problem of n classes, K words and so many levels may need: its
// list, that list's Q and P bits, the two bit strings a push makes, a frame per
// level (a level that finds no room for a list of its own works on the one
// above it with live bits of its own), and room for the keys of a leaf's L bits.
GMBE_HD long long cls_need(long long n, int K, int levels) {
  return cls_list_words(n, K) + 4 * cls_bit_words(n) + levels * cls_frame_words(n, K) + 512;
}
// Scratch of cls_build beside the list it makes: the masks before they have
// their places, bits and ranks of the candidates, the candidate of each mask
// (unless the caller has room for that elsewhere) and sums per vertex.
GMBE_HD long long cls_build_words(long long n, int K, bool own_mpos) {
  return cls_stride(n) * (K + (own_mpos ? 1 : 0)) + 4 * ((n + 63) >> 5) + 64;
}

// Words of the arena below a counts-tier push, for C candidates.  It holds any
// child of up to C classes, building and running: nothing a push makes is ever
// turned away for want of room.  Building, the most is the list, the masks, the
// candidate's C index (cls_stride) and the bits, 12 1/8 words a candidate with
// K = 4; running, the list and a bit per class and level, 11 1/8 words with 128
// levels, and 5,632 words of frames.
GMBE_HD long long cls_sub_words(long long C) { return 13 * C + 9696; }
// Words of keys and ids in front of a sub-problem that starts at a root or a slot.
GMBE_HD long long cls_key_words(int K) { return 96LL * K; }

}  // namespace gmbe
