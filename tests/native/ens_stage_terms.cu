// launch_ens_stage_sym (ens_stage.cu) with a term count that no kernel was built for: an error, and no
// CUDA call.  (No GPU needed.)
//
//   ens_stage_terms  ->  "refused N of M"
#include <cstdio>
#include <string>

#include "../../red.cuda.closeencounter_gb300/csrc/ens_stage.cu"

namespace redgb {
int set_error(int code, const std::string&) { return code; }
int cuda_fail(cudaError_t, const char*, const char*, int) { return RG_ERR_CUDA; }
}  // namespace redgb

int main()
{
    redgb::StageSymArgs a{};
    int refused = 0;
    const int counts[] = {-1, 0, 5, 10};
    for (int n : counts) refused += redgb::launch_ens_stage_sym(a, n, 1, nullptr) == RG_ERR_ARG;
    printf("refused %d of 4\n", refused);
    return refused == 4 ? 0 : 1;
}
