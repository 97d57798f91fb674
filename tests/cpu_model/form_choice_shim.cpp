// The choice between two forms of a solve (form_choice.cuh) for one host thread.
#include "form_choice.cuh"

extern "C" {
long long shim_attempts(double k, int n_out) { return dscb::attempts_estimate(k, n_out); }
int shim_short_chain_wins(int n, const double* k, int n_out, int limit)
{
    return dscb::short_chain_wins(dscb::HostTeam(), n, k, n_out, limit);
}
// bit 0: short chain, bit 1: many modes; gate
int shim_choice(int n_modes, long long limit, int* gate)
{
    const dscb::FormChoice c(n_modes, limit);
    *gate = c.gate();
    return (c.short_chain ? 1 : 0) | (c.many_modes ? 2 : 0);
}
}
