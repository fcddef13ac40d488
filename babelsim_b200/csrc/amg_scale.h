// Choice of the AMG coarse-correction scale from trial solves (KrylovSolver::tuneCorrection).  No device code.
#pragma once

#include <initializer_list>
#include <limits>

namespace bsg {

// A hierarchy that gains this much in a trial converges fast enough as it is (1e-10 in about 50).
constexpr double kTrialGood = 3e-5;
// What a trial reports that broke down or left no finite residual: worse than any that ran.
constexpr double kTrialFailed = std::numeric_limits<double>::infinity();

// The scale to use, given trial(scale, enough): the factor by which a trial reduced its residual; it may stop
// once that is `enough` (0: never).  `start` stays where it is good, or where no other does better.
template <class F>
double chooseCorrection(double start, F trial) {
    double chosen = start, best = trial(start, kTrialGood);
    if (best <= kTrialGood) return start;
    for (const double scale : {1.2, 1.5}) {
        const double reduced = trial(scale, 0.0);
        if (reduced < best) {
            best = reduced;
            chosen = scale;
        }
    }
    return chosen;
}

}  // namespace bsg
