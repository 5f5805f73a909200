// fgpe_error.h -- the message that fgpe_last_error(NULL) returns.
#pragma once
#include <string>

namespace fgpe {
void set_last_error(const std::string& m);
}
