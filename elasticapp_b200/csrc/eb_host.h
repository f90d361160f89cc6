// Host-side helpers shared between the simulator (eb_capi.cu) and the server
// (serve.cu).
#pragma once

#include <cstdint>
#include <string>

#include "../../include/elastica_b200.h"
#include "eb_internal.h"
#include "rod_init.h"

namespace eb {

// A straight rod's initializer (the checks of its arguments, and the part of
// its initial data that is computed once a rod; rod_init.cu has the rest)
eb_status straight_rod_spec(const eb_straight_rod& p, RodSpec& out);

// records the message eb_last_error() returns on this thread
void set_last_error(const std::string& message);

}  // namespace eb
