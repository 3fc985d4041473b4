// contact_flags.h — the words in which the detections of a contact phase raise
// "some vertex hit a face" (k_contact_phase).
//
// Detection n sets hit_word(n), a barrier follows, every CTA reads it, and
// thread 0 clears cleared_word(n).  A detection can follow the one before with
// no barrier in between (the Jacobi iterations have converged and a vertex
// still hits), so up to the next barrier the word being cleared may be neither
// the one being read (hit_word(n)) nor the one the next detection sets
// (hit_word(n + 1)): three words in turn.
#pragma once

namespace dfem {

constexpr int kHitWords = 3;
constexpr int hit_word(int n) { return n % kHitWords; }
constexpr int cleared_word(int n) { return (n + 2) % kHitWords; }

}  // namespace dfem
