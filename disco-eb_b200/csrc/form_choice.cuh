// Which of two forms of a solve takes a launch: the one with the shorter chain per mode (a block of
// warps, or one direction's) or the one with more modes in flight.
//
// The first lasts as long as its work, sum(attempts) / SMs; the second, while its modes are all in
// flight, as long as its longest mode.  So what decides is the work in lengths of the longest mode,
// sum(attempts) / max(attempts), which the number of modes bounds from above: up to `limit` modes the
// short chain wins whatever their wavenumbers.  In between, the kernels of both forms are launched, and
// each reads the wavenumbers, which are in device memory, and leaves if it is not its turn (some 5 us
// for 3000 wavenumbers, of solves of 30 ms and more).  The number of modes alone does not tell: 1536 modes
// of 72 rows from 1e-4 to 5 take 63.9 ms as blocks and 98.4 a warp each, from 1 to 5 155.2 and 114.9.
#pragma once

#include <cstdint>
#include <cstring>

#include "dual.cuh"
#include "team.cuh"

namespace dscb {

struct FormChoice {
    int limit;  // the work, in modes of the longest one's length, up to which the short chain wins
    bool short_chain, many_modes;  // the forms to launch
    // (log-spaced modes up to k = 10 are a quarter of the longest on the average, up to 5 a third, up to
    // 0.2 two thirds: above four times the limit the wavenumbers are not asked)
    FormChoice(int n_modes, long long lim)
        : limit(lim < 0x7fffffffLL ? (int)lim : 0x7fffffff), short_chain(n_modes <= 4 * lim), many_modes(n_modes > lim)
    {
    }
    // what the kernels get: the limit they compare the wavenumbers with, or kOnly
    int gate() const { return short_chain && many_modes ? limit : kOnly; }
    static constexpr int kOnly = -1;
};

// in a mode's status after the short chain's kernel has left the launch to the other form's
constexpr int32_t kOtherForm = -1;

// Tenths of step attempts of a mode, for their ratios: the counts of P(k) solves at rtol 1e-5 (70 at
// k = 6e-5 / Mpc, 357 at 0.016, 450 at 1, 1410 at 10), linear within an octave of k, and a third of an
// attempt per output time.  In integers, so that every kernel of a launch finds the same sum.
struct Attempts {
    int lo, hi, at[21];  // k = 2^lo .. 2^hi
};
#if defined(__CUDACC__)
static __device__  // (not constant memory, which serves a warp's different entries one after the other)
#endif
const Attempts kAttempts = {-14, 6, {70,  83,  103, 124, 145, 207, 272,  337,  357,  353, 348,
                                     347, 353, 362, 450, 709, 1000, 1290, 1784, 2520, 3570}};
DDV int64_t attempts_estimate(double k, int n_out)
{
    const Attempts& A = kAttempts;
#if defined(__CUDA_ARCH__)
    const uint64_t bits = (uint64_t)__double_as_longlong(k);
#else
    uint64_t bits;
    std::memcpy(&bits, &k, sizeof bits);
#endif
    int e = (int)((bits >> 52) & 0x7ff) - 1023, part = (int)((bits >> 40) & 0xfff);  // 2^e (1 + part / 4096)
    if (e < A.lo) { e = A.lo; part = 0; }
    if (e >= A.hi) { e = A.hi - 1; part = 4096; }
    const int i = e - A.lo;
    return 10 * (A.at[i] + (A.at[i + 1] - A.at[i]) * part / 4096) + 3 * (int64_t)n_out;
}

// whether the launch's modes are within `limit` lengths of the longest (every lane gets the answer)
template <class TM>
DDV bool short_chain_wins(const TM& tm, int n_modes, const double* kmodes, int n_out, int limit)
{
    int64_t sum = 0, longest = 0;
    for (int i = tm.lane; i < n_modes; i += TM::nl) {
        const int64_t a = attempts_estimate(kmodes[i], n_out);
        sum += a;
        longest = a > longest ? a : longest;
    }
#if defined(__CUDA_ARCH__)
    for (int o = 16; o > 0; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const int64_t other = __shfl_xor_sync(0xffffffffu, longest, o);
        longest = other > longest ? other : longest;
    }
#endif
    return sum <= longest * limit;
}

}  // namespace dscb
