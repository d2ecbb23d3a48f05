// The eigensolver's threads per CTA (khp_teams.h) for the CPU tests.
#include "khp_teams.h"

extern "C" {
int host_eig_team(int fp64, int n, int tuned) { return khp::eig_team(fp64 != 0, n, tuned); }
int host_chase_team(int n, long long batch, int tuned) { return khp::chase_team(n, batch, tuned); }
}
