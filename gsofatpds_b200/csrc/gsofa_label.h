// gsofa_label.h -- the word that label_cluster_kernel (gsofa_hub.cu) keeps per
// id: its label and, in bit 0, whether the id is idle (not queued).
//
// An expansion marks an id idle and must see every label given to it before; an
// improvement must queue the id unless a queued expansion will still see it.
// With the label and the mark in two words that needs sequentially consistent
// fences on both sides: the expansion's read could pass its clearing of the
// mark, while the improvement still finds the mark set.  In one word each side
// is a single atomic operation, and the order that all operations on one
// address have is enough:
//     expansion    word |= 1;            the value before holds the label to use
//     improvement  word = min(word, w);  queues the id iff the value before was
//                                        larger than w and idle
// A queued word is one less than the idle word of the same label, so a minimum
// with an equal label may queue the id once more; never once less.
#pragma once
#ifndef __CUDACC__
#define GSOFA_HD
#else
#define GSOFA_HD __host__ __device__ __forceinline__
#endif

namespace gsofa {

constexpr int kNoLabelWord = 0x7fffffff;  // no label yet, idle; its label is above every id below 2^30

// the word of an id that is queued with this label
GSOFA_HD constexpr int label_queued(int label) { return label << 1; }
GSOFA_HD constexpr int label_of_word(int word) { return word >> 1; }
// the bit an expansion sets
constexpr int kLabelIdle = 1;
// whether an improvement to `word` that found `before` queues the id
GSOFA_HD constexpr bool label_queues(int before, int word) { return before > word && (before & kLabelIdle); }

}  // namespace gsofa
