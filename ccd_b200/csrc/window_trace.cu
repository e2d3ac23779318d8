// window_trace.cu -- the windowed sweep with a stamp a round (CCDB_TRACE_FILE).
#define CCDB_TRACE_ROUNDS
#include "window.cu"
