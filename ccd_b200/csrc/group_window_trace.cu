// group_window_trace.cu -- the group models' windowed sweep with a stamp a round
// (CCDB_TRACE_FILE).
#define CCDB_TRACE_ROUNDS
#include "group_window.cu"
