// fixed_tables.hpp -- host side of the fixed-point tables (fixed_math.hpp).
#pragma once

#include "fixed_math.hpp"

namespace mcdg {

// The tables, computed at the first call in the process (thread-safe).
const FixedTables& fixed_tables();

}  // namespace mcdg
