// The download pool of the library over a counting stand-in for page-locked memory, for the CPU tests.
#include <atomic>
#include <cstdlib>

#include "../nuka-physics_b200/csrc/nkb_host_pool.h"

namespace {
std::atomic<long> g_locks{0}, g_unlocks{0}, g_live{0};
std::atomic<bool> g_refuse{false};

// no test writes to a block: large ones are address space only
void* Lock(size_t bytes) {
    if (g_refuse) return nullptr;
    ++g_locks; ++g_live;
    return std::malloc(bytes);
}
void Unlock(void* p) { ++g_unlocks; --g_live; std::free(p); }
}  // namespace

extern "C" {
void* pool_new() { return new nkb::HostPool(Lock, Unlock); }
void pool_delete(void* pool) { delete static_cast<nkb::HostPool*>(pool); }
void* pool_take(void* pool, size_t bytes) { return static_cast<nkb::HostPool*>(pool)->Take(bytes); }
void pool_give(void* pool, void* p) { static_cast<nkb::HostPool*>(pool)->Give(p); }
void pool_join(void* pool) { static_cast<nkb::HostPool*>(pool)->Join(); }
void pool_leave(void* pool) { static_cast<nkb::HostPool*>(pool)->Leave(); }
void pool_refuse(int on) { g_refuse = on != 0; }
long pool_locks() { return g_locks; }
long pool_unlocks() { return g_unlocks; }
long pool_live() { return g_live; }
}
