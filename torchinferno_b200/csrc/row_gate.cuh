// Rows multiplied by a gate, with an RMS norm ahead of it or behind it, 16 bytes a load (row_gate.cu).
#pragma once

#include "common.cuh"

namespace tib {

enum RowGate : int {
  ROW_GATE_ONLY = 0,      // x * sigmoid(z), z one number per column or per run of `group` columns
  ROW_GATE_LAST = 1,      // x / rms(x) * weight * sigmoid(z)
  ROW_GATE_FIRST = 2,     // v / rms(v) * weight with v = x * silu(z)
};

struct RowGateArgs {
  const void* x; int x_dtype; int64_t ldx;
  const void* z; int z_dtype; int64_t ldz;      // first column of the gate, row stride
  const float* weight;                          // [width], null for ROW_GATE_ONLY
  float eps;
  void* out; int out_dtype;                     // [rows, width]
  int rows, width, part, group;                 // the norm's mean is taken over each run of `part` columns
};

bool row_gate_takes(const RowGateArgs& a, int mode);
int row_gate(const RowGateArgs& a, int mode, cudaStream_t stream);

}  // namespace tib
