// The FP64 tensor instruction of the condensation, the standard element's
// tangent and the fronts.
#pragma once

namespace sbk {

// d += a (8 x 4, row-major) b (4 x 8): lane l holds a[l / 4][l % 4],
// b[l % 4][l / 4] and d[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void mma884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

}  // namespace sbk
