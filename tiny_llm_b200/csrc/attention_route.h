// Which launch of the 32-bit paged attention (attention_generic.cu) a step takes.  All give the same bits; only the time
// differs.  Plain C++, no CUDA.
#pragma once

namespace tllm {

// Rows per CTA of the kernel whose rows share their keys: 16 or 4, or 0 for the launches with a CTA or a warp per row (eight
// warps per row up to 8 rows per SM, one warp per four rows of a token above).
//   tokens, longest, requests   tokens of the step, the most of one request, requests (0: not known)
//   keys                        the most keys that a token of the step sees (an upper bound is fine; 0: not known)
//   nq, nk                      query and key rows of a token (heads times score maps)
//   wide                        rows of more than 64 values
// The lines, us per launch on a B200 (148 SMs), the kernel with shared rows / the other launches:
//   few keys            A CTA has 3.7 us behind it when its first tile is there, and is alone on its SM.  One wave (32 query
//                       over 4 key rows of 64): 9 keys 8.2 / 7.5, 13 8.9 / 8.9, 20 8.9 / 10.4, 100 8.2 / 13.7.  Barely
//                       more than a wave: 17 tokens of 32 heads of 128 with keys of their own, 17 keys 20 / 12, 48 20 / 16;
//                       33 tokens of 20 over 4 of 64 14 / 18.  64 decoded tokens: 31 keys 32 / 23, 48 29 / 33, 255 34 / 142.
//   several requests    in one CTA are walked one after the other.  Where a token's rows fill whole CTAs, or the requests
//                       bring many rows, none has several.  Two at a time (decoded tokens with groups of 2, 3, 5, 6, 7) cost
//                       what the other launch does while there are few requests (64 values: 37 / 35 at two to four requests
//                       with 700 keys, 128 values 55 / 42) and less with more of them, which share no fetch there (16
//                       requests: 37 / 53 and 55 / 79; with 40 keys 15 / 14 and 21 / 16).  Four at a time (a head with
//                       keys of its own): 68 / 36 at four requests with 700 keys beside 20 prompt tokens, 216 / 206 at 16
//                       with 1,400 beside 4.
//   many pairs          With more than 8 rows per SM the other launch walks a row's tiles in one warp: 64 tokens with 2,000
//                       keys 2,282, here 150.
inline int attention_rows_per_cta(long long tokens, long long longest, long long requests, long long keys, int nq, int nk,
                                  bool wide, int sms) {
  const long long group = nq / nk, pairs = tokens * nq, ctas = (tokens * group + 3) / 4 * nk;
  const long long others = tokens - longest, other_requests = requests > 1 ? requests - 1 : others;
  if (longest * group < 4) return 0;      // fewer than four rows share their keys
  const bool several = group % 4 != 0 && others > 0 && others * group < 8 * other_requests;
  if (pairs <= 8LL * sms) {
    if (keys > 0 && (keys <= 16 || (keys <= 48 && ctas > sms && pairs <= (wide ? 5LL : 4LL) * sms))) return 0;
    if (several && (group == 1 || 3 * others * nq <= 4LL * sms || (keys > 0 && keys <= 64))) return 0;
    return 4;
  }
  if (keys > 0 && keys <= (several ? 48 : 32)) return 0;
  // 16 rows where that gives every SM a CTA; with fewer CTAs half of the SMs would idle and a CTA's chain be longer
  return longest * group >= 16 && (tokens * group + 15) / 16 * nk >= sms ? 16 : 4;
}

}  // namespace tllm
