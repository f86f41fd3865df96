// Attention over few query rows (fa_split_sm100.cu); arguments are validated by the caller.
#pragma once

#include "host_common.h"

namespace hb {

bool fa_split_takes(const hb_fa_args* a, int sm_count);
uint64_t fa_split_workspace(const hb_fa_args* a, int sm_count);
int fa_split_run(const hb_fa_args* a, const DeviceState* st, void* workspace, uint64_t workspace_bytes);

}  // namespace hb
