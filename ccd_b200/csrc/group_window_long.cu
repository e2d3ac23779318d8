// group_window_long.cu -- the group models' windowed sweep for Cox fits with long columns.
#define CCDB_COX_LONG
#include "group_window.cu"
