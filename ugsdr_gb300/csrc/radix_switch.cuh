// One switch per pass to code with the radix compiled in.
#pragma once

#include <type_traits>

namespace ugsdr_gpu {

	// calls fn(integral_constant<int, R>) for R = r, 2 <= r <= MAXR <= 32
	template <int MAXR, class Fn>
	__device__ __forceinline__ void with_radix(int r, Fn&& fn) {
#define UG_RADIX(R)                                     \
	case R:                                             \
		if constexpr (R <= MAXR)                        \
			fn(std::integral_constant<int, R>{});       \
		break;
		switch (r) {
			UG_RADIX(2) UG_RADIX(3) UG_RADIX(4) UG_RADIX(5) UG_RADIX(6) UG_RADIX(7) UG_RADIX(8) UG_RADIX(9)
			UG_RADIX(10) UG_RADIX(11) UG_RADIX(12) UG_RADIX(13) UG_RADIX(14) UG_RADIX(15) UG_RADIX(16) UG_RADIX(17)
			UG_RADIX(18) UG_RADIX(19) UG_RADIX(20) UG_RADIX(21) UG_RADIX(22) UG_RADIX(23) UG_RADIX(24) UG_RADIX(25)
			UG_RADIX(26) UG_RADIX(27) UG_RADIX(28) UG_RADIX(29) UG_RADIX(30) UG_RADIX(31) UG_RADIX(32)
		}
#undef UG_RADIX
	}
}
