// Exchange of tridiag_reg.cu: which words a CTA of the cluster waits for in a step.
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
// CTAs past the eighth get no share: warp w sends CTA kWarps + w a zero (-1: none).
AGB_HD int zero_dest(int w, int Ce) { return kWarps + w < Ce ? kWarps + w : -1; }
// Words that CTA q gets from each CTA, and their pitch at the receiver.
AGB_HD int dot_words(int q, int Ce) { return q < kWarps ? (kWarps - q + Ce - 1) / Ce : 1; }
AGB_HD int dot_pitch(int Ce) { return (kWarps + Ce - 1) / Ce; }

// Columns of a CTA's slice (a multiple of cpt, the columns of a thread).
AGB_HD int slice(int n, int Ce, int cpt) { return ((n + Ce - 1) / Ce + cpt - 1) / cpt * cpt; }

// Bytes that CTA q waits for in step j on barrier 1 (V owners of rows) and barrier 2.
AGB_HD int bytes1(int n, int Ce, int V, int cpt, int q, int j) {
  const int S = slice(n, Ce, cpt);
  const int used = (j + 1) / cpt * cpt;  // columns below it are finished, cpt at a time
  const int first = q * S > used ? q * S : used, end = n < q * S + S ? n : q * S + S;
  const int groups = end > first ? (end - first + cpt - 1) / cpt : 0;
  return groups * (V + 1) * cpt * 8 + dot_words(q, Ce) * Ce * 4;
}
AGB_HD int bytes2(int n, int Ce, int j) { return (n - 1 - j) * 16 + Ce * 4; }

}  // namespace exchange
