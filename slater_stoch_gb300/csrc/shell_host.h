// shell_host.h -- host entry points of the shell-quartet path (shell_tables.cu) and the side
// streams it shares with the per-function kernels (ss_api.cu).
#pragma once
#include <vector>

#include "ss_context.cuh"

namespace ss {

// work entries by total degree
struct ShellPlan {
  std::vector<ShWork> work[SH_MAXL + 1];
};

int shell_precond(ss_ctx* c, std::vector<double>& pre);
int shell_plan(ss_ctx* c, bool tiers, const std::vector<int64_t>& sel, std::vector<int64_t>& slot, std::vector<int64_t>& rest,
               ShellPlan& plan, int64_t* nelem);
int shell_run(ss_ctx* c, ShellPlan& plan, double eps, double eps32, double* elem);

// the side streams start after everything queued on the context stream; the context stream waits
// for all of them
int fork_eri_streams(ss_ctx* c);
int join_eri_streams(ss_ctx* c);

}  // namespace ss
