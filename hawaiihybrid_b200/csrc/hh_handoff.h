// The tuner's choice of the hand-off threshold, (multiple / divisor) x the solo kernel's warp
// slots, from timed launches.  Host code, free of CUDA, so that the rule can be tested with
// made-up times.
#pragma once

namespace hh {
constexpr int HANDOFF_MUL_MAX = 8;  // largest multiple
constexpr int HANDOFF_DIV_MAX = 4;  // largest divisor (with multiple 1)
// A candidate has to be faster than the choice so far by this factor.  Two runs of one
// threshold differ by up to 1 %, neighbouring ones by 0 to 10 %: taken as soon as it is faster
// at all, from the smallest multiple up and stopping at the first that is not, three of eight
// tunings of CO2-Ar (FP64, 20,000 x 4,096) left a threshold 5 % slower than the default for the
// life of the context.
constexpr float HANDOFF_GAIN = 0.98f;

// run(div, mul, &ms): 0 and the launch's time, or an error, which ends the choice.  Starts at
// multiple `def`, goes to larger ones while each is faster, and if none is, to smaller ones.
template <class Run> int pick_handoff(int def, const Run &run, int *div, int *mul) {
  float best = 0.f, t = 0.f;
  *div = 1;
  *mul = def;
  int rc = run(1, def, &best);
  if (rc) return rc;
  auto take = [&](int d, int m, bool *better) {
    const int e = run(d, m, &t);
    *better = !e && t < HANDOFF_GAIN * best;
    if (*better) {
      best = t;
      *div = d;
      *mul = m;
    }
    return e;
  };
  bool better = true;
  for (int m = 2 * def; m <= HANDOFF_MUL_MAX && better; m *= 2)
    if ((rc = take(1, m, &better))) return rc;
  if (*mul != def) return 0;
  better = true;
  for (int m = def / 2; m >= 1 && better; m /= 2)
    if ((rc = take(1, m, &better))) return rc;
  if (*mul > 1) return 0;
  better = true;
  for (int d = 2; d <= HANDOFF_DIV_MAX && better; d *= 2)
    if ((rc = take(d, 1, &better))) return rc;
  return 0;
}
}  // namespace hh
