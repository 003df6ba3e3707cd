// decode_token_kernel instantiations for YALM_F16 weights.
#include "decode_token.cuh"

namespace yalm {
namespace mega {
const void *kernel_f16_token(int head_dim, int g) {
	set_fault_pointers(fault_record(), fault_timeout_cycles() > 0 ? fault_timeout_cycles() : token::kPatience);
	return token::token_kernel_for<YALM_F16>(head_dim, g);
}
} // namespace mega
} // namespace yalm
