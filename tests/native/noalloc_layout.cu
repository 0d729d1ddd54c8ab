// Where the engine's counters hold a job's error word.
#include <cstddef>

#include "iwpp_engine.cuh"

extern "C" size_t engine_ctrl_bytes() { return sizeof(iwpp::Ctrl); }
extern "C" size_t engine_ctrl_error_at() { return offsetof(iwpp::Ctrl, error); }
