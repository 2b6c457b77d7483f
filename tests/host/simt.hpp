// Runs device code of the library on the CPU: every GPU thread is a fiber,
// warps exchange through __shfl_*_sync, CTAs meet in __syncthreads and
// clusters in this_cluster().sync().  A fiber runs until it has to wait.
//
// Fibers are scheduled by priority: all CTAs of lower rank go as far as they
// can before a higher rank starts (or the reverse), the least favourable
// order for a cluster.  An access to the shared memory of a CTA that has not
// started, or has ended, is counted.  Shared memory starts as 0xFF bytes
// (NaN), so a read before the first write shows.
//
// Include before the library's headers; compiled by the host compiler alone.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <setjmp.h>
#include <string.h>
#include <ucontext.h>

#include <functional>
#include <memory>
#include <vector>

namespace simt {

struct Barrier {
  int need = 0, here = 0;
  long gen = 0;
  bool any = false, last_any = false;  // of the arrivals, and of the last round
};
struct Fiber {
  ucontext_t ctx;  // its first entry; later switches by jumps, which make no system call
  jmp_buf at;
  bool begun = false;
  std::unique_ptr<char[]> stack;
  int tid = 0, rank = 0;
  Barrier *wait = nullptr;
  long gen = 0;
  bool done = false;
};
struct Warp {
  Barrier bar;
  double slot[2][32];
  int flip[32] = {};
};
struct Cta {
  Barrier bar;
  std::vector<Warp> warps;
  std::vector<unsigned char> smem;
  bool started = false;
  int left = 0;
};
struct Machine {
  jmp_buf home;
  std::vector<Fiber> fibers;
  std::vector<Cta> ctas;
  Barrier cluster;
  Fiber *cur = nullptr;
  int nt = 0;
  long early = 0;  // accesses to a CTA that has not started or has ended
  std::function<void()> body;
};
inline Machine *m = nullptr;

inline void block(Barrier &b)  // arrives; returns when all have
{
  if (++b.here == b.need) {
    b.here = 0;
    b.last_any = b.any;
    b.any = false;
    b.gen++;
    return;
  }
  Fiber *f = m->cur;
  f->wait = &b;
  f->gen = b.gen;
  if (!_setjmp(f->at)) _longjmp(m->home, 1);
}
inline Cta &cta() { return m->ctas[m->cur->rank]; }
inline void entry()
{
  m->body();
  m->cur->done = true;
  cta().left--;
  _longjmp(m->home, 1);
}
inline __attribute__((noinline)) void resume(Fiber &f)
{
  if (_setjmp(m->home)) return;
  if (f.begun) _longjmp(f.at, 1);
  f.begun = true;
  setcontext(&f.ctx);
}
// One cluster of cn CTAs (cn = 1: a plain CTA) of nt threads with `bytes` of
// shared memory each; returns the number of accesses to CTAs not running, or
// -1 if some fiber waits for good.
inline long run(int cn, int nt, size_t bytes, bool high_first, std::function<void()> body)
{
  Machine mm;
  m = &mm;
  mm.nt = nt;
  mm.body = body;
  mm.ctas.resize(cn);
  mm.cluster.need = cn * nt;
  for (Cta &c : mm.ctas) {
    c.bar.need = c.left = nt;
    c.smem.assign(bytes + 16, 0xff);
    c.warps.resize(nt / 32);
    for (Warp &w : c.warps) w.bar.need = 32;
  }
  mm.fibers.resize((size_t)cn * nt);
  for (int i = 0; i < cn * nt; i++) {
    Fiber &f = mm.fibers[i];
    f.rank = high_first ? cn - 1 - i / nt : i / nt;
    f.tid = i % nt;
    f.stack.reset(new char[64 * 1024]);
    getcontext(&f.ctx);
    f.ctx.uc_stack.ss_sp = f.stack.get();
    f.ctx.uc_stack.ss_size = 64 * 1024;
    f.ctx.uc_link = nullptr;
    makecontext(&f.ctx, entry, 0);
  }
  for (;;) {
    int left = 0;
    bool ran = false;
    for (int r = 0; r < cn && !ran; r++)  // the first CTA of the order that can run
      for (int i = r * nt; i < (r + 1) * nt; i++) {
        Fiber &f = mm.fibers[i];
        if (f.done) continue;
        left++;
        if (f.wait && f.wait->gen == f.gen) continue;
        f.wait = nullptr;
        mm.cur = &f;
        mm.ctas[f.rank].started = true;
        resume(f);
        ran = true;
      }
    if (!ran) {
      m = nullptr;
      return left ? -1 : mm.early;
    }
  }
}
template <class T> T *shared() { return reinterpret_cast<T *>(((uintptr_t)cta().smem.data() + 15) & ~(uintptr_t)15); }

template <class T> T shfl(T x, int src)  // one rendezvous: the slots alternate
{
  Warp &w = cta().warps[m->cur->tid >> 5];
  const int lane = m->cur->tid & 31, f = w.flip[lane];
  w.flip[lane] ^= 1;
  memcpy(&w.slot[f][lane], &x, sizeof(T));
  block(w.bar);
  T y;
  memcpy(&y, &w.slot[f][src], sizeof(T));
  return y;
}

struct Dim {
  struct X {
    operator int() const { return m->cur->tid; }
  } x;
};
struct BDim {
  struct X {
    operator int() const { return m->cur->rank; }
  } x;
};
struct NDim {
  struct X {
    operator int() const { return m->nt; }
  } x;
};

}  // namespace simt

#undef __shared__
#define __shared__ static  // one CTA at a time
#define threadIdx (simt::Dim())
#define blockIdx (simt::BDim())
#define blockDim (simt::NDim())
template <class T> T __shfl_xor_sync(unsigned, T x, int o) { return simt::shfl(x, (simt::m->cur->tid & 31) ^ o); }
template <class T> T __shfl_sync(unsigned, T x, int s) { return simt::shfl(x, s & 31); }
inline int __any_sync(unsigned, int p)
{
  int any = 0;
  for (int o = 0; o < 32; o++) any |= simt::shfl(p, o);
  return any;
}
inline void __syncwarp() { simt::block(simt::cta().warps[simt::m->cur->tid >> 5].bar); }
inline void __syncthreads() { simt::block(simt::cta().bar); }
inline int __syncthreads_or(int p)
{
  simt::Barrier &b = simt::cta().bar;
  b.any = b.any || p;
  simt::block(b);
  return b.last_any;
}
inline int __clz(int x) { return x ? __builtin_clz((unsigned)x) : 32; }
template <class T> T min(T a, T b) { return b < a ? b : a; }
template <class T> T max(T a, T b) { return a < b ? b : a; }

namespace cooperative_groups {
struct Cluster {
  void sync() const { simt::block(simt::m->cluster); }
  template <class T> T *map_shared_rank(T *p, int q) const
  {
    simt::Cta &c = simt::m->ctas[q];
    if (!c.started || c.left == 0) simt::m->early++;
    const size_t off = reinterpret_cast<unsigned char *>(p) - simt::cta().smem.data();
    // same offset from the aligned base, whatever the vectors' addresses
    const size_t mine = reinterpret_cast<unsigned char *>(simt::shared<unsigned char>()) - simt::cta().smem.data();
    unsigned char *base = reinterpret_cast<unsigned char *>(((uintptr_t)c.smem.data() + 15) & ~(uintptr_t)15);
    return reinterpret_cast<T *>(base + (off - mine));
  }
};
inline Cluster this_cluster() { return {}; }
}  // namespace cooperative_groups
