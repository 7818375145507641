// The words of BatchArgs::st that a solve's first CTA leaves for every CTA of
// k_batch32, four per solve (plain C++, so that the rule can be checked on a host).
#pragma once

#ifdef __CUDACC__
#define NSS_HD __host__ __device__
#else
#define NSS_HD
#endif

namespace nss {

// st[0], st[1] of a step: alpha and h_j, written before the step's second
// barrier and read after it, before the next step's first one.
constexpr int ST_ALPHA = 0, ST_HJ = 1, ST_WORDS = 4;

// The projections that a solve still asks for after step k: written at the end
// of step k, read after the second barrier of step k + 1.  A step that does not
// project has no barrier behind that read, so step k + 1 must not write the
// word that a slower CTA may still be reading: the steps take two words in
// turn.  The next write of a word, at the end of step k + 2, has the barriers of
// step k + 2 before it.
NSS_HD constexpr int owed_word(int step) { return 2 + (step & 1); }

}  // namespace nss
