// Test infrastructure, not product code: the routes by size
// (mercury_b200/csrc/routes.h) behind a C interface.
#include "../mercury_b200/csrc/routes.h"

extern "C" {
int triangle_route(int64_t n, int64_t nnz) { return (int)mc::triangle_route_by_size(n, nnz); }
int pattern_route(int64_t n, int64_t nnz, int64_t max_degree, int pattern) {
  return (int)mc::pattern_route_by_size(n, nnz, max_degree, pattern);
}
int samples(int64_t n, int64_t nnz, int64_t max_degree, int pattern) {
  return mc::probe_percent(n, nnz, max_degree, pattern);
}
int batch_bits(int64_t n, int64_t nnz, int64_t max_degree, int64_t squares, int pattern) {
  return (int)mc::batch_takes_bits(n, nnz, max_degree, squares, pattern);
}
}
