// A warp on the CPU: 32 fibers run the same code and meet at every warp collective, so code
// written for one warp (dds_gpu_b200/csrc/ddg_warp.cuh) runs and is checked without a GPU.
//
// The fibers take turns in a ring. A collective leaves its operand in this fiber's slot and
// yields; when the turn comes back every other fiber has left its own (two sets of slots in
// turn, since a fiber may reach the next collective before the others have read this one).
// Every collective also leaves its kind: fibers that meet at different ones are an error.
#pragma once
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include <vector>

extern "C" void emu_switch(void** save_sp, void* to_sp);
asm(R"(
.text
.globl emu_switch
.type emu_switch, @function
emu_switch:
  pushq %rbp
  pushq %rbx
  pushq %r12
  pushq %r13
  pushq %r14
  pushq %r15
  movq %rsp, (%rdi)
  movq %rsi, %rsp
  popq %r15
  popq %r14
  popq %r13
  popq %r12
  popq %rbx
  popq %rbp
  ret
.size emu_switch, .-emu_switch
)");

struct WarpEmu {
  enum { LANES = 32, STACK = 256 * 1024 };
  void* sp[LANES];
  void* host_sp = nullptr;
  std::vector<char> stacks;
  uint32_t val[2][LANES];
  int kind[2][LANES];
  unsigned turn[LANES];  // collectives this fiber has reached
  int cur = 0, left = 0;
  bool backwards = false;  // the ring's direction: which fibers run ahead of which
  void (*body)(void*, int) = nullptr;
  void* arg = nullptr;
  static thread_local WarpEmu* self;

  static void entry() {
    WarpEmu* e = self;
    e->body(e->arg, e->cur);
    if (--e->left) e->yield(true);
    void* dummy;
    emu_switch(&dummy, e->host_sp);  // the last fiber hands back to the host
    abort();
  }
  void yield(bool done = false) {
    const int me = cur;
    if (done) sp[me] = nullptr;
    int next = me;
    do {
      next = (next + (backwards ? LANES - 1 : 1)) % LANES;
    } while (!sp[next] && next != me);
    cur = next;
    void* ignore;
    emu_switch(done ? &ignore : &sp[me], sp[next]);
  }
  void run(void (*f)(void*, int), void* a) {
    body = f;
    arg = a;
    self = this;
    stacks.resize((size_t)LANES * STACK);
    for (int t = 0; t < LANES; t++) {
      uintptr_t top = ((uintptr_t)stacks.data() + (size_t)(t + 1) * STACK) & ~(uintptr_t)15;
      void** s = (void**)top;
      *--s = nullptr;  // keeps the stack 16-byte aligned at entry
      *--s = (void*)&WarpEmu::entry;
      for (int k = 0; k < 6; k++) *--s = nullptr;
      sp[t] = s;
      turn[t] = 0;
    }
    left = LANES;
    cur = 0;
    emu_switch(&host_sp, sp[0]);
  }
  const uint32_t* meet(int what, uint32_t v) {
    const int me = cur, set = turn[me]++ & 1;
    val[set][me] = v;
    kind[set][me] = what;
    yield();
    for (int t = 0; t < LANES; t++)
      if (kind[set][t] != what) {
        fprintf(stderr, "warp emulation: fiber %d is at collective %d, fiber %d at %d\n", me, what, t, kind[set][t]);
        abort();
      }
    return val[set];
  }
};
thread_local WarpEmu* WarpEmu::self = nullptr;

static inline uint32_t w_ballot(bool p) {
  const uint32_t* v = WarpEmu::self->meet(1, p);
  uint32_t m = 0;
  for (int t = 0; t < 32; t++) m |= (uint32_t)(v[t] != 0) << t;
  return m;
}
static inline uint32_t w_shfl(uint32_t x, int src) { return WarpEmu::self->meet(2, x)[src & 31]; }
static inline uint32_t w_shfl_up1(uint32_t x) {
  const int me = WarpEmu::self->cur;
  return WarpEmu::self->meet(3, x)[me ? me - 1 : 0];
}
static inline uint32_t w_or(uint32_t x) {
  const uint32_t* v = WarpEmu::self->meet(4, x);
  uint32_t r = 0;
  for (int t = 0; t < 32; t++) r |= v[t];
  return r;
}
static inline uint32_t w_max(uint32_t x) {
  const uint32_t* v = WarpEmu::self->meet(5, x);
  uint32_t r = 0;
  for (int t = 0; t < 32; t++) r = v[t] > r ? v[t] : r;
  return r;
}
static inline uint32_t w_min(uint32_t x) {
  const uint32_t* v = WarpEmu::self->meet(6, x);
  uint32_t r = 0xFFFFFFFFu;
  for (int t = 0; t < 32; t++) r = v[t] < r ? v[t] : r;
  return r;
}
static inline uint32_t w_add(uint32_t x) {
  const uint32_t* v = WarpEmu::self->meet(7, x);
  uint32_t r = 0;
  for (int t = 0; t < 32; t++) r += v[t];
  return r;
}
static inline void w_sync() { WarpEmu::self->meet(8, 0); }
