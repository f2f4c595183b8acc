// Exchange of tridiag_reg.cu: the words of v^H A v that the CTAs of a cluster send.
// Host code too: tests/test_tridiag_exchange.py compiles this file by itself.
//
// Barrier 1 collects a CTA's partial p's and the next row over its column slice, and
// words of v^H A v; barrier 2 the reduced columns and one word of every CTA.  A CTA
// whose slice is used up has nothing but the words to wait for on barrier 1, and
// what it sends next counts on its peers' barrier 2.  So it waits there for a word
// of EVERY peer: a peer sends that one after its own barrier 2 of the previous step,
// and no byte of a step can then reach a barrier that still counts the step before.
#pragma once
#ifndef AGB_HD
#define AGB_HD inline
#endif

namespace exchange {

constexpr int kWarps = 8;  // per CTA; clusters have at most 2 kWarps CTAs

// Warp w's share of v^H A v goes to CTA w mod Ce.
AGB_HD int dot_dest(int w, int Ce) { return w % Ce; }
// CTAs past the eighth get no share but a zero: CTA kWarps + w, from warp w below this.
AGB_HD int zeros(int Ce) { return Ce > kWarps ? Ce - kWarps : 0; }
// Words that CTA q gets, and waits for, from each CTA; their pitch at the receiver.
AGB_HD int dot_words(int q, int Ce) { return q < kWarps ? (kWarps - q + Ce - 1) / Ce : 1; }
AGB_HD int dot_pitch(int Ce) { return (kWarps + Ce - 1) / Ce; }

}  // namespace exchange
