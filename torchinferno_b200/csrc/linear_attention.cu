// Linear attention with a fixed decay per head over per-request state:
//     S_t = lambda * S_(t-1) + k_t v_t^T        (S: [key_dim, value_dim], fp32, one per request, layer call and head)
//     o_t = S_t^T q_t
// for the tokens of a ragged batch: portions of prompts and single decoded tokens alike.  An optional
// activation (silu) is applied to q, k and v as they are read, in fp32.
//
// One block owns one (request entry, head, run of value columns): the columns of S do not depend on one another, so
// a head is cut into runs of columns that go to blocks of their own until the grid fills the GPU (each recomputes the
// chunk's scores, which are cheap beside the state).  A block keeps its columns of S in shared memory and walks the
// entry's tokens in chunks of up to C: within a chunk of n tokens
//     A[i][j] = (q_i . k_j) lambda^(i-j)                                    j <= i
//     o_i     = lambda^(i+1) S^T q_i + sum_(j<=i) A[i][j] v_j
//     S      <- lambda^n S + sum_j lambda^(n-1-j) k_j v_j^T
// which is the recurrence written out.  Scores, decay powers, state and sums are fp32; the powers
// lambda^0 .. lambda^C come from the host as a table (made in double precision).  A single token is a chunk
// of one.  State is read from and written back to the request's slot; a new request's slot is zero.
//
// Three ways to run that.  Every portion takes the one its own length and the layer's sizes name, whatever else is in the step
// (tib_linear_attention launches each form that occurs over the whole batch, and a form's blocks leave the others' portions alone), so a
// request's numbers do not depend on its neighbours:
//   runs   (portions above 192 tokens, or 384 in heads of 64 x 64; head sizes of 64 or 128) every run of 128 tokens makes its own sum L of decayed k v^T
//          side by side, one thread per state element then folds S <- lambda^n S + L over a request's runs, and every run
//          makes its outputs from its starting state: the serial chain is one fused multiply-add a run
//   walk   (portions of at most 32 tokens) S in registers, token by token
//   chunks (everything else) the block walk described above
#include "linear_attention.cuh"

namespace tib {

struct LinAttnArgs {
  const int* q_start;     // [n_entries + 1]
  const int* slots;       // [n_entries]
  const float* powers;    // [heads, chunk + 1]
  float* state;           // [slots, heads, key_dim, value_dim]
  float* out;             // [tokens, heads * value_dim]
  int64_t ldq, ldk, ldv;  // row strides of q, k, v (elements)
  int heads, key_dim, value_dim, chunk, activation;
  int cols;               // value columns per block
  int shortest, longest;  // the portions this launch takes (the others are another form's)
};

template <typename T>
__global__ void __launch_bounds__(256)
linear_attention_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, LinAttnArgs a) {
  extern __shared__ float smem[];
  const int D = a.key_dim, C = a.chunk, DP = D + 1;
  const int col0 = blockIdx.z * a.cols;
  const int V = min(a.cols, a.value_dim - col0);       // this block's columns: col0 .. col0 + V - 1 of the head's value_dim
  float* S = smem;                 // [D][V]
  float* qs = S + D * a.cols;      // [C][DP]
  float* ks = qs + C * DP;         // [C][DP]
  float* vs = ks + C * DP;         // [C][V], on a 16-byte boundary (rows of four columns are read as one)
  vs += (4 - (int)((vs - smem) & 3)) & 3;
  float* A = vs + C * a.cols;      // [C][C]
  float* pw = A + C * C;           // [C + 1]
  const int head = blockIdx.x, entry = blockIdx.y;
  pdl_wait();
  pdl_trigger();
  const int row0 = a.q_start[entry], len = a.q_start[entry + 1] - row0;
  if (len < a.shortest || len > a.longest) return;
  float* state = a.state + ((size_t)a.slots[entry] * a.heads + head) * D * a.value_dim + col0;      // row stride value_dim
  for (int e = threadIdx.x; e < D * V; e += blockDim.x) S[e] = state[(size_t)(e / V) * a.value_dim + e % V];
  for (int e = threadIdx.x; e <= C; e += blockDim.x) pw[e] = a.powers[head * (C + 1) + e];

  // bf16 rows on 16-byte boundaries are fetched eight elements a load, and the next chunk's rows are asked for before
  // the current chunk is worked on (they wait in registers): fetched element by element where they were needed, the
  // rows cost a chain of memory latencies per chunk, more than the arithmetic.
  constexpr int kPieces = 4;       // 16-byte pieces a thread holds per tensor
  const int dp = D / 8, vp = V / 8;
  bool wide = false;
  if constexpr (sizeof(T) == 2) {
    wide = D % 8 == 0 && V % 8 == 0 && col0 % 8 == 0 && a.value_dim % 8 == 0 && a.ldq % 8 == 0 && a.ldk % 8 == 0 && a.ldv % 8 == 0 &&
           ((uintptr_t)q & 15) == 0 && ((uintptr_t)k & 15) == 0 && ((uintptr_t)v & 15) == 0 &&
           C * dp <= kPieces * (int)blockDim.x && C * vp <= kPieces * (int)blockDim.x;
  }
  uint4 rq[kPieces], rk[kPieces], rv[kPieces];
  auto ask = [&](int t0) {
    const int n = min(C, len - t0);
#pragma unroll
    for (int it = 0; it < kPieces; ++it) {
      const int p = threadIdx.x + it * blockDim.x;
      if (p < n * dp) {
        const int i = p / dp, c = (p - i * dp) * 8;
        const size_t row = row0 + t0 + i;
        rq[it] = *reinterpret_cast<const uint4*>(q + row * a.ldq + head * D + c);
        rk[it] = *reinterpret_cast<const uint4*>(k + row * a.ldk + head * D + c);
      }
      if (p < n * vp) {
        const int i = p / vp, c = (p - i * vp) * 8;
        rv[it] = *reinterpret_cast<const uint4*>(v + (size_t)(row0 + t0 + i) * a.ldv + head * a.value_dim + col0 + c);
      }
    }
  };
  auto unpack = [&](const uint4& raw, float* dst) {
    const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const float2 f = bf16x2_floats(h2[x]);
      dst[2 * x] = lin_act(f.x, a.activation);
      dst[2 * x + 1] = lin_act(f.y, a.activation);
    }
  };
  if (wide) ask(0);

  for (int t0 = 0; t0 < len; t0 += C) {
    const int n = min(C, len - t0);
    __syncthreads();               // the chunk before is done with qs, ks, vs, A (and S, pw are loaded)
    if (wide) {
#pragma unroll
      for (int it = 0; it < kPieces; ++it) {
        const int p = threadIdx.x + it * blockDim.x;
        if (p < n * dp) {
          const int i = p / dp, c = (p - i * dp) * 8;
          unpack(rq[it], qs + i * DP + c);
          unpack(rk[it], ks + i * DP + c);
        }
        if (p < n * vp) {
          const int i = p / vp, c = (p - i * vp) * 8;
          unpack(rv[it], vs + i * V + c);
        }
      }
      if (t0 + C < len) ask(t0 + C);
    } else {
      for (int e = threadIdx.x; e < n * D; e += blockDim.x) {
        const int i = e / D, d = e - i * D;
        const size_t row = row0 + t0 + i;
        qs[i * DP + d] = lin_act(to_f32(q[row * a.ldq + head * D + d]), a.activation);
        ks[i * DP + d] = lin_act(to_f32(k[row * a.ldk + head * D + d]), a.activation);
      }
      for (int e = threadIdx.x; e < n * V; e += blockDim.x) {
        const int i = e / V, c = e - i * V;
        vs[i * V + c] = lin_act(to_f32(v[(size_t)(row0 + t0 + i) * a.ldv + head * a.value_dim + col0 + c]), a.activation);
      }
    }
    __syncthreads();
    // scores: a thread takes a 2 x 2 block (rows i, i + 1; keys j, j + 1), so four products share four loads
    {
      const int half = (n + 1) / 2;
      for (int e = threadIdx.x; e < half * half; e += blockDim.x) {
        const int bi = e / half, bj = e - bi * half;
        const int i = 2 * bi, j = 2 * bj;
        if (j > i + 1) continue;                       // the block lies above the diagonal
        const int i1 = min(i + 1, n - 1), j1 = min(j + 1, n - 1);
        float s00 = 0.f, s01 = 0.f, s10 = 0.f, s11 = 0.f;
        for (int d = 0; d < D; ++d) {
          const float q0 = qs[i * DP + d], q1 = qs[i1 * DP + d], k0 = ks[j * DP + d], k1 = ks[j1 * DP + d];
          s00 = fmaf(q0, k0, s00); s01 = fmaf(q0, k1, s01); s10 = fmaf(q1, k0, s10); s11 = fmaf(q1, k1, s11);
        }
        A[i * C + j] = j <= i ? s00 * pw[i - j] : 0.f;
        if (j + 1 < n) A[i * C + j + 1] = j + 1 <= i ? s01 * pw[i - j - 1] : 0.f;
        if (i + 1 < n) {
          A[(i + 1) * C + j] = s10 * pw[i + 1 - j];
          if (j + 1 < n) A[(i + 1) * C + j + 1] = j + 1 <= i + 1 ? s11 * pw[i - j] : 0.f;
        }
      }
    }
    __syncthreads();
    if ((V & 3) == 0) {
      // outputs and state: a thread takes four neighbouring columns (one 16-byte load of S or v per step)
      const int V4 = V >> 2;
      for (int e = threadIdx.x; e < n * V4; e += blockDim.x) {
        const int i = e / V4, c = (e - i * V4) * 4;
        float4 carried = make_float4(0.f, 0.f, 0.f, 0.f), inside = carried;
        for (int d = 0; d < D; ++d) {
          const float qv = qs[i * DP + d];
          const float4 sv = *reinterpret_cast<const float4*>(S + d * V + c);
          carried.x = fmaf(qv, sv.x, carried.x); carried.y = fmaf(qv, sv.y, carried.y);
          carried.z = fmaf(qv, sv.z, carried.z); carried.w = fmaf(qv, sv.w, carried.w);
        }
        for (int j = 0; j <= i; ++j) {
          const float av = A[i * C + j];
          const float4 vv = *reinterpret_cast<const float4*>(vs + j * V + c);
          inside.x = fmaf(av, vv.x, inside.x); inside.y = fmaf(av, vv.y, inside.y);
          inside.z = fmaf(av, vv.z, inside.z); inside.w = fmaf(av, vv.w, inside.w);
        }
        float* dst = a.out + (size_t)(row0 + t0 + i) * a.heads * a.value_dim + head * a.value_dim + col0 + c;
        const float pi = pw[i + 1];
        dst[0] = fmaf(pi, carried.x, inside.x); dst[1] = fmaf(pi, carried.y, inside.y);
        dst[2] = fmaf(pi, carried.z, inside.z); dst[3] = fmaf(pi, carried.w, inside.w);
      }
      __syncthreads();               // every o of the chunk has read the old S
      for (int e = threadIdx.x; e < D * V4; e += blockDim.x) {
        const int d = e / V4, c = (e - d * V4) * 4;
        float4 add = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j = 0; j < n; ++j) {
          const float kv = pw[n - 1 - j] * ks[j * DP + d];
          const float4 vv = *reinterpret_cast<const float4*>(vs + j * V + c);
          add.x = fmaf(kv, vv.x, add.x); add.y = fmaf(kv, vv.y, add.y); add.z = fmaf(kv, vv.z, add.z); add.w = fmaf(kv, vv.w, add.w);
        }
        float4* sp = reinterpret_cast<float4*>(S + d * V + c);
        float4 sv = *sp;
        const float pn = pw[n];
        sv.x = fmaf(pn, sv.x, add.x); sv.y = fmaf(pn, sv.y, add.y); sv.z = fmaf(pn, sv.z, add.z); sv.w = fmaf(pn, sv.w, add.w);
        *sp = sv;
      }
    } else {
      for (int e = threadIdx.x; e < n * V; e += blockDim.x) {
        const int i = e / V, c = e - i * V;
        float carried = 0.f, inside = 0.f;
        for (int d = 0; d < D; ++d) carried = fmaf(qs[i * DP + d], S[d * V + c], carried);
        for (int j = 0; j <= i; ++j) inside = fmaf(A[i * C + j], vs[j * V + c], inside);
        a.out[(size_t)(row0 + t0 + i) * a.heads * a.value_dim + head * a.value_dim + col0 + c] = fmaf(pw[i + 1], carried, inside);
      }
      __syncthreads();               // every o of the chunk has read the old S
      for (int e = threadIdx.x; e < D * V; e += blockDim.x) {
        const int d = e / V, c = e - d * V;
        float add = 0.f;
        for (int j = 0; j < n; ++j) add = fmaf(pw[n - 1 - j] * ks[j * DP + d], vs[j * V + c], add);
        S[e] = fmaf(pw[n], S[e], add);
      }
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < D * V; e += blockDim.x) state[(size_t)(e / V) * a.value_dim + e % V] = S[e];
}

// ---------------------------------------------------------------------------------------------------------- runs
// The walk above is one serial chain of 64 chunks for 2,048 tokens, each with four barriers, on 512 blocks that each see 32 of a
// run's 128 columns: 980 us for two portions of 1,366 and 682 tokens, 16 heads of 128 x 128, of which the fp32 arithmetic
// (3.3 GFLOP here) is some 50 us.  In runs of 64 on the fp32 pipe the three launches took 131 us in the layer (one by one and cold 49 + 27 + 82); in
// runs of 128 on the tensor cores (linear_tcgen05.cu) they take 68 (cold 22 + 16 + 44), half of the states' traffic with it.  Of 2,048 tokens of 24 heads of 64 x 64
// 57 us (74), of 600 of 8 heads of 128 x 64 27 (33).
// Everything stays fp32 or three bf16 terms of it: activations, decay powers, scores, states and sums.  Error against 64 bits (2-norm, those
// four cases with one of 4 heads of 64 x 128): outputs 1.0 to 1.3e-7 (1.4 to 1.9 on the fp32 pipe), states 7 to 8.7e-8 (8.6e-8 to 1.0e-7).
// The shortest portion that is cut into runs (why: tib_linear_attention).
static int lin_runs_from(int key_dim, int value_dim) { return key_dim * value_dim <= 64 * 64 ? 385 : 193; }
// grid (state elements / 1024, entries): S <- lambda^n S + L over the entry's runs, four elements a thread; run_state turns from
// a run's sum into the state at its start, the last state goes to the slot.
__global__ void __launch_bounds__(256) lin_fold_kernel(LinRunArgs a, int key_dim) {
  pdl_wait();
  pdl_trigger();
  const int entry = blockIdx.y, row0 = a.q_start[entry], len = a.q_start[entry + 1] - row0;
  const size_t per_head = (size_t)key_dim * a.value_dim, width = per_head * a.n_heads;
  const size_t e = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;
  if (len < a.shortest || e >= width) return;
  const float* pw = a.powers + (a.head0 + e / per_head) * (kLinRun + 1);
  const int runs = (len + kLinRun - 1) / kLinRun, last = len - (runs - 1) * kLinRun;
  const float whole = pw[kLinRun], part = pw[last];
  float* run = a.run_state + lin_first_run(row0, entry) * width + e;
  float4* slot = reinterpret_cast<float4*>(a.state + ((size_t)a.slots[entry] * a.heads + a.head0) * per_head + e);
  float4 st = *slot;
  constexpr int AHEAD = 8;      // (loads in flight a thread: the fold is a chain of memory latencies)
  for (int r = 0; r < runs; r += AHEAD) {
    float4 sum[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (r + u < runs) sum[u] = *reinterpret_cast<const float4*>(run + (size_t)(r + u) * width);
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      if (r + u >= runs) break;
      *reinterpret_cast<float4*>(run + (size_t)(r + u) * width) = st;
      const float f = r + u == runs - 1 ? part : whole;
      st = make_float4(fmaf(f, st.x, sum[u].x), fmaf(f, st.y, sum[u].y), fmaf(f, st.z, sum[u].z), fmaf(f, st.w, sum[u].w));
    }
  }
  *slot = st;
}

// ---------------------------------------------------------------------------------------------------------- walk
// Single tokens and portions of a few: a block holds 32 columns of one head's S in registers (a thread four neighbouring columns
// of every 32nd row), so a step reads and writes the state once, 16 bytes a load with all of a thread's loads in flight.
// What bounds it is the launch and one trip to memory: eight tokens of 16 heads of 128 x 128 8 us (cold), 42 in the chunk kernel,
// whose score is one thread's chain of 128 products for a single token.
constexpr int kLinWalk = 32;            // the longest portion it takes
constexpr int kLinWalkStage = 8;        // tokens it holds in shared memory at a time

template <typename T, int ROWS>         // ROWS: key_dim / 32
__global__ void __launch_bounds__(256)
lin_walk_kernel(const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, LinRunArgs a) {
  constexpr int D = ROWS * 32;
  constexpr int C = kLinWalkStage;
  __shared__ float qs[C][D], ks[C][D];
  __shared__ __align__(16) float vs[C][32];
  __shared__ float4 red[C][8][8];
  pdl_wait();
  pdl_trigger();
  const int tiles = a.value_dim / 32, head = blockIdx.x / tiles, col0 = (blockIdx.x - head * tiles) * 32;
  const int entry = blockIdx.y, row0 = a.q_start[entry], len = a.q_start[entry + 1] - row0;
  if (len <= 0 || len > kLinWalk) return;
  const int tid = threadIdx.x, cg = tid & 7, rt = tid >> 3;
  float* S = a.state + ((size_t)a.slots[entry] * a.heads + head) * (size_t)D * a.value_dim + col0 + cg * 4;
  float4 s[ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) s[i] = *reinterpret_cast<const float4*>(S + (size_t)(rt + 32 * i) * a.value_dim);
  const float lambda = a.powers[head * (kLinRun + 1) + 1];
  for (int t0 = 0; t0 < len; t0 += C) {
    const int n = min(C, len - t0);
    const size_t first = row0 + t0;
    for (int e = tid; e < n * D; e += 256) {
      const int t = e / D, d = e % D;
      qs[t][d] = lin_act(to_f32(q[(first + t) * a.ldq + head * D + d]), a.activation);
      ks[t][d] = lin_act(to_f32(k[(first + t) * a.ldk + head * D + d]), a.activation);
    }
    if (tid < n * 32)
      vs[tid >> 5][tid & 31] = lin_act(to_f32(v[(first + (tid >> 5)) * a.ldv + head * a.value_dim + col0 + (tid & 31)]), a.activation);
    __syncthreads();
    for (int t = 0; t < n; ++t) {
      const float4 vv = *reinterpret_cast<const float4*>(&vs[t][cg * 4]);
      float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < ROWS; ++i) {
        const float kk = ks[t][rt + 32 * i], qq = qs[t][rt + 32 * i];
        s[i] = make_float4(fmaf(lambda, s[i].x, kk * vv.x), fmaf(lambda, s[i].y, kk * vv.y), fmaf(lambda, s[i].z, kk * vv.z),
                           fmaf(lambda, s[i].w, kk * vv.w));
        o.x = fmaf(qq, s[i].x, o.x); o.y = fmaf(qq, s[i].y, o.y); o.z = fmaf(qq, s[i].z, o.z); o.w = fmaf(qq, s[i].w, o.w);
      }
#pragma unroll
      for (int m = 8; m < 32; m <<= 1) {
        o.x += __shfl_xor_sync(0xffffffffu, o.x, m); o.y += __shfl_xor_sync(0xffffffffu, o.y, m);
        o.z += __shfl_xor_sync(0xffffffffu, o.z, m); o.w += __shfl_xor_sync(0xffffffffu, o.w, m);
      }
      if ((tid & 31) < 8) red[t][tid >> 5][cg] = o;
    }
    __syncthreads();               // the partial sums are in place, and q, k, v of these tokens no longer needed
    if (tid < n * 8) {
      const int t = tid >> 3;
      float4 o = red[t][0][cg];
#pragma unroll
      for (int w = 1; w < 8; ++w) {
        const float4 p = red[t][w][cg];
        o.x += p.x; o.y += p.y; o.z += p.z; o.w += p.w;
      }
      *reinterpret_cast<float4*>(a.out + (first + t) * a.heads * a.value_dim + head * a.value_dim + col0 + cg * 4) = o;
    }
    // (the next tokens' partial sums are written only after the barrier behind their loads, which the threads above reach last)
  }
#pragma unroll
  for (int i = 0; i < ROWS; ++i) *reinterpret_cast<float4*>(S + (size_t)(rt + 32 * i) * a.value_dim) = s[i];
}

static int launch_lin_runs(const void* q, const void* k, const void* v, const LinRunArgs& a, int dtype, int key_dim, int n_entries, int max_q_len,
                           cudaStream_t stream) {
  const int runs = ceil_div(max_q_len, kLinRun);
  // Tiles of 128 value columns, or of 64 where those leave half of the SMs without one.
  const int tile = a.value_dim % 128 == 0 && (int64_t)a.n_heads * (a.value_dim / 128) * runs * n_entries > 74 ? 128 : 64;
  const dim3 grid(a.n_heads * (a.value_dim / tile), runs, n_entries);
  int status = launch_lin_run_sums(k, v, a, dtype, key_dim, tile, grid, stream);
  if (status != TIB_OK) return status;
  TIB_LAUNCH_DEPENDENT(lin_fold_kernel, dim3((unsigned)ceil_div64((int64_t)a.n_heads * key_dim * a.value_dim, 1024), n_entries), 256, 0, stream, a, key_dim);
  return launch_lin_run_outs(q, k, v, a, dtype, key_dim, tile, grid, stream);
}

template <typename T>
static int launch_lin_walk(const void* q, const void* k, const void* v, const LinRunArgs& a, int key_dim, int n_entries, cudaStream_t stream) {
  const dim3 grid(a.heads * (a.value_dim / 32), n_entries);
  if (key_dim == 64) TIB_LAUNCH_DEPENDENT((lin_walk_kernel<T, 2>), grid, 256, 0, stream, (const T*)q, (const T*)k, (const T*)v, a);
  else TIB_LAUNCH_DEPENDENT((lin_walk_kernel<T, 4>), grid, 256, 0, stream, (const T*)q, (const T*)k, (const T*)v, a);
  return TIB_OK;
}

static inline size_t lin_attn_smem(int D, int V, int C) {
  return sizeof(float) * ((size_t)D * V + 2 * (size_t)C * (D + 1) + 3 + (size_t)C * V + (size_t)C * C + C + 1);
}

}  // namespace tib

using namespace tib;

// The largest chunk (32, 16, 8, 4, 2 or 1 tokens) whose working set fits an SM's shared memory; 0 if none does.
TIB_API int tib_linear_attention_chunk(int key_dim, int value_dim) {
  for (int c = 32; c >= 1; c >>= 1)
    if (lin_attn_smem(key_dim, value_dim, c) <= 227 * 1024) return c;
  return 0;
}

// Tokens of a run, the longest portion the walk takes, and the shortest that is cut into runs in heads of these sizes.
TIB_API int tib_linear_attention_run() { return kLinRun; }
TIB_API int tib_linear_attention_walk() { return kLinWalk; }
TIB_API int tib_linear_attention_runs_from(int key_dim, int value_dim) { return lin_runs_from(key_dim, value_dim); }

// q, k: [tokens, >= heads * key_dim] and v: [tokens, >= heads * value_dim] with row strides ldq, ldk, ldv (they may be
// slices of one wider row); out: [tokens, heads * value_dim] fp32; state: [slots, heads, key_dim, value_dim] fp32;
// powers: [heads, chunk + 1] fp32, powers[h][m] = lambda_h^m; activation: 0 none, 1 silu on q, k and v.
// forms: which portions occur, 1: of at most tib_linear_attention_walk() tokens, 4: of tib_linear_attention_runs_from() and more, 2:
// between them; 0 where it is not known (then, or without run_powers, the chunk kernel runs them all).  n_chunked: how many portions lie
// between them (at most; the chunk kernel shares a head's columns out by it).  max_q_len: the longest portion.
// run_powers: [heads, run + 1] fp32 likewise, or null.  run_state: scratch of run_capacity >= tokens / run + n_entries times
// run_heads * key_dim * value_dim floats for portions of tib_linear_attention_runs_from() tokens and more, which are worked run_heads heads
// at a time, or null (they run in chunks then).
// launches: takes the number of kernels launched.
TIB_API int tib_linear_attention(const void* q, const void* k, const void* v, int64_t ldq, int64_t ldk, int64_t ldv,
                                 float* out, float* state, const float* powers, const int* q_start, const int* slots,
                                 int n_entries, int heads, int key_dim, int value_dim, int chunk, int activation, int dtype,
                                 int tokens, int max_q_len, int forms, int n_chunked, const float* run_powers, float* run_state, int64_t run_capacity, int run_heads,
                                 int* launches, int* error_word, cudaStream_t stream) {
  *launches = 0;
  if (n_entries == 0) return TIB_OK;
  if (!q || !k || !v || !out || !state || !powers || !q_start || !slots) return TIB_E_ARG;
  if (heads < 1 || key_dim < 1 || value_dim < 1 || chunk < 1 || chunk > 32 || n_entries > 65535) return TIB_E_SIZE;
  // The newer kernels take heads of 64 or 128 keys whose values come in whole tiles, rows and state on 16-byte boundaries.
  // The lines between the three.  Walk and chunks (four portions of 16 heads of 128 x 128): 14, 16 and 23 us at 8, 9 and 16 tokens
  // against 33, 33 and 35.  Chunks and runs, the whole layer's device time at 40 / 64 / 128 / 192 tokens: one portion of 16 heads of 128 x 128
  // 36 / 41 / 66 / 91 us against 37 / 37 / 39 / 41, four of them 69 / 86 / 152 / 221 against 45 / 47 / 56 / 71; one portion of 12 heads of 64 x 64
  // 24 / 25 / 39 / 52 against 28 / 28 / 30 / 30.  On the device alone the lines would lie near 50 tokens.  But a prompt's layer is issued call by
  // call, which takes 81 us of the host in chunks and 91 in runs (two launches and an allocation more), and what is shorter on the device than
  // that waits for the host.  Call by call, a lone portion in chunks and in runs: 128 x 128 84 and 91 at 160 tokens, 96 and 91 at 192, 121
  // and 91 at 256; 64 x 64 82 and 91 at 256, 97 and 91 at 384.  Several portions would gain from 64 tokens on, and not know of it: the line
  // goes by a portion's own length.
  const int64_t size = dtype == TIB_F32 ? 4 : 2;
  const bool aligned = (ldq * size) % 16 == 0 && (ldk * size) % 16 == 0 && (ldv * size) % 16 == 0 &&
                       (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)state | (uintptr_t)out | (uintptr_t)run_state) & 15) == 0;
  int shortest = 1;      // what is left for the chunk kernel
  int longest = 0x7fffffff, chunked = n_entries;
  if (run_powers && forms && (key_dim == 64 || key_dim == 128) && value_dim % 32 == 0 && aligned && (dtype == TIB_F32 || dtype == TIB_BF16)) {
    LinRunArgs r;
    r.q_start = q_start; r.slots = slots; r.powers = run_powers; r.state = state; r.run_state = run_state; r.out = out;
    r.ldq = ldq; r.ldk = ldk; r.ldv = ldv; r.heads = heads; r.head0 = 0; r.n_heads = heads; r.shortest = lin_runs_from(key_dim, value_dim); r.value_dim = value_dim; r.activation = activation;
    r.error_word = error_word;
    if (forms & 1) {
      const int status = dtype == TIB_F32 ? launch_lin_walk<float>(q, k, v, r, key_dim, n_entries, stream)
                                          : launch_lin_walk<__nv_bfloat16>(q, k, v, r, key_dim, n_entries, stream);
      if (status != TIB_OK) return status;
      *launches += 1;
    }
    shortest = kLinWalk + 1;
    const bool runs = run_state && run_heads > 0 && value_dim % 64 == 0 && run_capacity >= tokens / kLinRun + n_entries && ceil_div(max_q_len, kLinRun) <= 65535;
    if ((forms & 4) && runs) {
      for (; r.head0 < heads; r.head0 += run_heads) {
        r.n_heads = run_heads < heads - r.head0 ? run_heads : heads - r.head0;
        const int status = launch_lin_runs(q, k, v, r, dtype, key_dim, n_entries, max_q_len, stream);
        if (status != TIB_OK) return status;
        *launches += 3;
      }
    }
    if (runs) longest = r.shortest - 1;
    if (runs || !(forms & 4)) {
      if (!(forms & 2)) return TIB_OK;
      chunked = n_chunked > 0 && n_chunked < n_entries ? n_chunked : n_entries;
    }
  }
  LinAttnArgs a;
  a.shortest = shortest; a.longest = longest;
  a.q_start = q_start; a.slots = slots; a.powers = powers; a.state = state; a.out = out;
  a.ldq = ldq; a.ldk = ldk; a.ldv = ldv;
  a.heads = heads; a.key_dim = key_dim; a.value_dim = value_dim; a.chunk = chunk; a.activation = activation;
  // runs of value columns: halve them (down to 8) while the grid has fewer than two blocks per SM
  int cols = value_dim;
  while (cols >= 16 && cols % 2 == 0 && (int64_t)heads * chunked * (value_dim / cols) < 2 * 148) cols /= 2;
  a.cols = cols;
  const size_t smem = lin_attn_smem(key_dim, cols, chunk);
  if (smem > 227 * 1024) return TIB_E_SMEM;
  dim3 grid(heads, n_entries, ceil_div(value_dim, cols));
  if (dtype == TIB_F32) {
    auto kern = linear_attention_kernel<float>;
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem);
      if (e != cudaSuccess) return (int)e;
    }
    TIB_LAUNCH_DEPENDENT(kern, grid, 256, smem, stream, (const float*)q, (const float*)k, (const float*)v, a);
  } else if (dtype == TIB_BF16) {
    auto kern = linear_attention_kernel<__nv_bfloat16>;
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem);
      if (e != cudaSuccess) return (int)e;
    }
    TIB_LAUNCH_DEPENDENT(kern, grid, 256, smem, stream, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k,
                         (const __nv_bfloat16*)v, a);
  } else {
    return TIB_E_DTYPE;
  }
  *launches += 1;
  return TIB_OK;
}

// The calls the Python parts make (common.cuh).
TIB_PACKED(tib_linear_attention)
TIB_PACKED(tib_linear_attention_chunk)
TIB_PACKED(tib_linear_attention_run)
TIB_PACKED(tib_linear_attention_runs_from)
TIB_PACKED(tib_linear_attention_walk)
