// pair_shape.cu -- the search behind pair_shape.h (host arithmetic).
#include "pair_shape.h"

#include <math.h>

#include <algorithm>

namespace esrrf {

namespace {

// The shape with the least modelled time for `units` (strip, frame) pairs of H rows.  A segment also
// walks the 2R + 1 rows around it and costs about 8 rows to start and drain; the short ones run one
// after another with nothing beside them, about 25 rows more each (both measured).  An SM runs
// `maxw` warps (by their registers and shared memory); with w warps it reaches 1 - exp(-w / 8.5) of its full rate (measured
// at R = 6: 8 warps 0.7 of the rate of 16), and a second CTA on it costs 15 %, more of them 40 %: they
// fetch the taps' code apart.  CTAs of equal length go in waves; a last segment of another length fills the
// slots that the last wave of the long ones leaves free (33 frames of 512 x 512 at M4, 132 CTAs: 4.89
// ms with segments of 1863 + 185 rows, 5.13 with 1925 + 123).
PairShape pair_shape_search(int units, int H, int R, int maxw, int sms) {
    const double extra = 2 * R + 9, extra_last = extra + 25;
    PairShape best;
    for (int warps = maxw; warps >= 4; warps /= 2) {
        const int per_sm = maxw / warps, n1 = (units + warps - 1) / warps;
        const long slots = (long)sms * per_sm;
        auto rate = [&](int ctas) {  // time of one row on an SM with that many CTAs
            const double w = (double)ctas * warps;
            return w / (1.0 - exp(-w / 8.5)) * (1.0 + 0.15 * (ctas > 1) + 0.25 * (ctas > 2));
        };
        const double full = rate(per_sm);
        // time of n CTAs of `len` rows, all together
        auto waves = [&](long n, double len) {
            const long q = n / slots, r = n - q * slots;
            return len * (q * full + (r ? rate((int)((r + sms - 1) / sms)) : 0.0));
        };
        for (int k = 1; k <= 48 && (k == 1 || H / k >= 8); ++k) {
            const int even = (H + k - 1) / k;
            for (int part = 0; part < 11; ++part) {  // part 0: k equal segments; else shorter ones and a rest
                const int rows = part == 0 ? even : (int)(even * (1.0 - 0.015 * part));
                const int rest = H - k * rows;
                if (part && (rest < 8 || rows < 8)) continue;
                double t;
                if (rest <= 0) {
                    t = waves((long)n1 * k, rows + extra);
                } else {
                    // the short ones start in the slots that are free in the last wave of the long ones
                    const double tl = (rows + extra) * full, ts = (rest + extra_last) * full;
                    const long n = (long)n1 * k, q = n / slots, r = n - q * slots;
                    double end = q * tl;
                    for (long done = 0; done < n1; end += ts) {
                        done += slots - r;
                        if (end + ts >= (q + 1) * tl && r) done += r * (long)((end + ts - (q + 1) * tl) / ts);
                    }
                    t = std::max(end, (q + (r ? 1 : 0)) * tl);
                }
                if (best.cost == 0 || t < 0.99 * best.cost) {
                    best.warps = warps;
                    best.rows = rows;
                    best.segs = rest > 0 ? k : (H + rows - 1) / rows;
                    best.cost = t;
                }
            }
        }
    }
    return best;
}

}  // namespace

// The last few shapes of this thread (a block's launches have one or two sizes).
PairShape pair_shape(int units, int H, int R, int maxw, int sms) {
    struct Memo {
        int units = -1, H = 0, R = 0, maxw = 0, sms = 0;
        PairShape shape;
    };
    thread_local Memo memo[4];
    thread_local int next = 0;
    for (const Memo& m : memo)
        if (m.units == units && m.H == H && m.R == R && m.maxw == maxw && m.sms == sms) return m.shape;
    Memo& m = memo[next++ & 3];
    m.units = units, m.H = H, m.R = R, m.maxw = maxw, m.sms = sms;
    m.shape = pair_shape_search(units, H, R, maxw, sms);
    return m.shape;
}

}  // namespace esrrf
