// The FP64 tensor instruction, for the kernels that include this inside their anonymous namespaces.
#pragma once

// c (8 x 8; lane: row lane / 4, columns 2 (lane % 4), + 1) += a (8 x 4; row lane / 4, column lane % 4) b (4 x 8; row
// lane % 4, column lane / 4)
__device__ __forceinline__ void dmma884(double &c0, double &c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}
