// prompt_plan.cuh -- how many tokens the work buffers of a context's prompt passes hold (engine.cu).  Host code without CUDA, so that it is tested without a device.
#pragma once

#include <algorithm>

#define PIB_PROMPT_MAX 1024          // tokens per pass of the tensor-core prompt path (gemm_q4k_tc.cu)
#define PIB_PROMPT_STAGE 256         // the shortest buffers; and the passes where several stages work on one prompt: passes of the stages overlap

// Two sizes, so that a context allocates twice at most: PIB_PROMPT_STAGE until a prompt is longer, then PIB_PROMPT_MAX or what the context holds.  Larger buffers are made
// before the smaller ones go; what memory refused is not asked for again (an attempt costs allocations that synchronise the device), and the smaller ones stay in use.
struct pib_prompt_plan {
    int cap = 0;                     // tokens that the buffers hold
    int limit = PIB_PROMPT_MAX;      // the largest size that has not been refused
    int want(int n_tokens, int n_ctx, int stages) const {
        return stages > 1 || n_tokens <= PIB_PROMPT_STAGE ? PIB_PROMPT_STAGE : std::max(PIB_PROMPT_STAGE, std::min(limit, std::min(PIB_PROMPT_MAX, (n_ctx + 255) / 256 * 256)));
    }
    // make(n): allocates buffers for n tokens and puts them in the old ones' place, or changes nothing and returns false.  False: there are no buffers at all
    template <typename Make> bool grow(int n_tokens, int n_ctx, int stages, Make make) {
        for (int n = want(n_tokens, n_ctx, stages); n > cap; n -= 256) {
            if (make(n)) { cap = n; return true; }
            limit = std::max(PIB_PROMPT_STAGE, n - 256);
        }
        return cap > 0;
    }
};
