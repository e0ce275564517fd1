// Recurrences over a per-sequence float32 state, eight tokens at a time: see chunk_scan.cu.
#pragma once
#include <cuda_runtime.h>

enum ChunkScanKind {
    CHUNK_LINEAR = 0,       // S <- a S + k v^T, one fixed decay per head
    CHUNK_DELTA_HEAD = 1,   // the gated delta rule, a decay per head and token
    CHUNK_DELTA_CHANNEL = 2 // the same, a decay per head, key channel and token
};

struct ChunkScanArgs {
    const float *q, *k, *v;         // token t, query/key head hk: q + t * ld + hk * d; value head h: v + t * ld + h * dv
    long long ld;
    const float* g;                 // the decays: LINEAR [nh]; DELTA_HEAD [T, nh]; DELTA_CHANNEL [T, nh * d]
    const float* beta;              // the delta rule's write strengths [T, nh]
    int nh, share, d, dv;           // value head h reads query/key head h / share
    float* state;                   // slot s, head h: S as [dv][d] at state + slots * state_stride + h * d * dv
    long long state_stride;
    const int *slots, *cu_q;
    float* rec;                     // scratch: chunk_scan_scratch floats
    float* out;                     // [T, nh * dv]
    int segments;                   // LINEAR: pieces of a sequence that run side by side (1: in order)
    float* seg_state;               // [B, segments, nh, dv, d], with segments > 1
};

// Heads of up to 128 key channels, any value size.
inline bool chunk_scan_takes(int d) { return d >= 1 && d <= 128; }
long long chunk_scan_scratch(long long T, int B, int nh);
int chunk_scan_segments(int kind, int B, int nh, int dv, int max_q);
int chunk_scan_launch(const ChunkScanArgs& a, int kind, int B, int max_q, cudaStream_t s);
