// Several launches of one kernel as one.
//
// The per-element kernels of the mixed path run over buckets of wires (one Nk each) and over the
// matrices P, C, D; on small wires such a launch is a few us of latency and a few blocks.  Here the
// parts of one pass share a launch: each part has its own arguments and its own grid, a block
// finds its part and its place in that part's grid.
#pragma once
#include "launch.cuh"

namespace sbe {

// a block's place in its part: blockIdx, and the x extent of the part's grid
struct Blk {
  int x, y, z, gx;
};

template <class... T>
struct Args {};
template <class H, class... T>
struct Args<H, T...> {
  H h;
  Args<T...> t;
};

template <int N, class... P>
struct Parts {
  int n, same;                  // same: all parts have one gx, gy
  int first[N], gx[N], gy[N];   // first block, or first z of a common grid; extents of the grid
  Args<P...> a[N];
};

template <class Body, class... A>
__device__ __forceinline__ void call_part(const Blk& b, const Args<>&, const A&... a) {
  Body::run(b, a...);
}
template <class Body, class H, class... T, class... A>
__device__ __forceinline__ void call_part(const Blk& b, const Args<H, T...>& s, const A&... a) {
  call_part<Body>(b, s.t, a..., s.h);
}

template <class Body, int N, class... P>
__global__ void __launch_bounds__(Body::kThreads, Body::kBlocks)
    k_parts(const __grid_constant__ Parts<N, P...> p) {
  pdl_enter();
  const int at = p.same ? blockIdx.z : blockIdx.x;
  int i = 0;   // a constant with one part: its arguments stay where they are
  if constexpr (N > 1)
    while (i + 1 < p.n && at >= p.first[i + 1]) ++i;
  Blk b{(int)blockIdx.x, (int)blockIdx.y, at - p.first[i], (int)gridDim.x};
  if (!p.same) {
    const int gy = p.gy[i], row = b.z / p.gx[i];
    b.gx = p.gx[i];
    b.x = b.z - row * b.gx;
    b.y = row % gy;
    b.z = row / gy;
  }
  const Args<P...> a = p.a[i];
  call_part<Body>(b, a);
}

// Collects the parts of one pass and launches them, kMax a launch; a pass of few parts takes a
// small parameter block.  A sweep of 64 wires in seven buckets: 548 launches a step, 83 so (57 with
// the passes joined since), and 3.87 -> 2.27 ms (one launch per part left the SMs between a few small blocks and the launch
// gap); 1 x 64 (P, C, D together) 403 -> 334 us.
template <class Body, class F = decltype(Body::signature())>
class Batch;
template <class Body, class... P>
class Batch<Body, void (*)(Blk, P...)> {
 public:
  Batch(dim3 block, cudaStream_t s, size_t smem = 0) : block_(block), s_(s), part_smem_(smem) {}
  ~Batch() { flush(); }
  // dynamic shared memory of the parts that follow; a launch asks for its own parts' largest
  void smem(size_t bytes) { part_smem_ = bytes; }
  template <class... A>
  void add(dim3 grid, A&&... a) {
    const long long blocks = (long long)grid.x * grid.y * grid.z;
    if (blocks == 0) return;
    if (p_.n == kMax || blocks_ + blocks > 0x7fffffffLL) flush();
    const int i = p_.n++;
    smem_ = smem_ > part_smem_ ? smem_ : part_smem_;
    z_[i] = grid.z;
    p_.gx[i] = grid.x;
    p_.gy[i] = grid.y;
    set(p_.a[i], a...);
    blocks_ += blocks;
  }
  void flush() {
    if (p_.n == 0) return;
    // one Nk: a common grid, stacked in z, spares the blocks the divisions
    long long z = 0, flat = 0;
    p_.same = 1;
    for (int i = 0; i < p_.n; ++i) {
      p_.same = p_.same && p_.gx[i] == p_.gx[0] && p_.gy[i] == p_.gy[0];
      z += z_[i];
    }
    p_.same = p_.same && z <= 65535 && p_.gy[0] <= 65535;
    z = 0;
    for (int i = 0; i < p_.n; ++i) {
      p_.first[i] = (int)(p_.same ? z : flat);
      z += z_[i];
      flat += (long long)p_.gx[i] * p_.gy[i] * z_[i];
    }
    const dim3 grid = p_.same ? dim3(p_.gx[0], p_.gy[0], (unsigned)z) : dim3((unsigned)flat);
    if (p_.n == 1)
      start<1>(grid);
    else if (p_.n <= 4)
      start<4>(grid);
    else
      start<kMax>(grid);
    p_.n = 0;
    blocks_ = 0;
    smem_ = 0;
  }

 private:
  static constexpr int kMax = 24;
  template <int N>
  void start(dim3 grid) {
    Parts<N, P...> f{};
    f.n = p_.n;
    f.same = p_.same;
    for (int i = 0; i < p_.n; ++i) {
      f.first[i] = p_.first[i];
      f.gx[i] = p_.gx[i];
      f.gy[i] = p_.gy[i];
      f.a[i] = p_.a[i];
    }
    launch(k_parts<Body, N, P...>, grid, block_, smem_, s_, f);
  }
  static void set(Args<>&) {}
  template <class H, class... T, class A, class... B>
  static void set(Args<H, T...>& d, A&& a, B&&... b) {
    d.h = static_cast<H>(a);
    set(d.t, b...);
  }
  Parts<kMax, P...> p_{};
  long long blocks_ = 0;
  int z_[kMax] = {};
  dim3 block_;
  cudaStream_t s_;
  size_t smem_ = 0, part_smem_;
};

// Names a device function, void(Blk, ...), as the body of a batched pass (blocks: per SM at least,
// 0 for no bound).
#define SBE_PASS_BLOCKS(Name, threads, blocks, ...)             \
  struct Name {                                                 \
    static constexpr int kThreads = threads, kBlocks = blocks;  \
    static decltype(&__VA_ARGS__) signature();                  \
    template <class... A>                                       \
    __device__ __forceinline__ static void run(const A&... a) { \
      __VA_ARGS__(a...);                                        \
    }                                                           \
  }
#define SBE_PASS(Name, threads, ...) SBE_PASS_BLOCKS(Name, threads, 0, __VA_ARGS__)

}  // namespace sbe
