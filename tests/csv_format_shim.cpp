// Test infrastructure: the CSV writer's cells (yallasql_b200/csrc/yq_csv.cuh)
// compiled for the host with g++, so the CPU suite can compare the longest text
// of every type with the bound that the writer's callers allocate by.
#include "../yallasql_b200/csrc/yq_csv.cuh"

using namespace yq::csv;

extern "C" {

int32_t hs_max_cell(int32_t type, int32_t width) { return max_cell(type, width); }

// One cell's text into `out` (no NUL); returns its length as CountOut has it, -1 when BufOut disagrees.
int32_t hs_format_cell(const void* data, const uint8_t* nulls, int32_t type, int32_t width, uint64_t row,
                       uint8_t* out) {
  CountOut n;
  put_cell(n, data, nulls, type, width, row);
  BufOut o{out};
  put_cell(o, data, nulls, type, width, row);
  return (uint32_t)(o.p - out) == n.n ? (int32_t)n.n : -1;
}

}  // extern "C"
