// Internal runtime services shared by the entry points.
#pragma once

#include <cstddef>
#include <mutex>

#include "sigma_common.h"

namespace sigma {

// Serialises the host-pointer entry points (they share cached buffers).
std::mutex& api_mutex();

// Multiprocessor count of the current device (0 when no device).
int device_sm_count();

// Grow-only device buffers of the current device, one per slot; freed by
// sigma_shutdown().  The caller holds api_mutex().
constexpr int kArenaSlots = 6;
enum ArenaSlot {
  kArenaGppInputs = 0,
  kArenaFfInputs = 1,
  kArenaBatched = 2,
  kArenaMisc = 3,
  kArenaExact = 4,     // contraction workspaces of host calls' plans
  kArenaExactOcc = 5
};
int arena_get(int slot, size_t bytes, void** out);
// An optional workspace of a plan that lives for one host call, up to 256 MB
// kept between calls (allocating and freeing one costs the small calls 130 us);
// null above that or without room.  drop_optional_arenas frees them; no plan
// may be using one.
void* arena_optional(int slot, size_t bytes);
void drop_optional_arenas();

// Whether an optional workspace may be taken: it leaves at least as much of
// the current device's free memory as it takes (up to 256 MB without asking:
// the question takes 80 us).
bool room_for_optional(size_t bytes);

// Functions that give back the optional workspaces of plan caches; run (and
// the allocation tried again) when an arena, or a host call's plan, finds no
// memory.  The caller holds api_mutex().
typedef void (*ReclaimHook)();
void register_reclaim_hook(ReclaimHook h);
void reclaim_caches();

// A host call's plan (create returns a status), and its arena beside the
// plan's own optional workspace (drop gives it up).
template <class F>
int with_reclaim(F create) {
  const int st = create();
  if (st != SIGMA_ERR_ALLOC) return st;
  reclaim_caches();
  drop_optional_arenas();
  return create();
}
template <class F>
int arena_beside(int slot, size_t bytes, void** out, F drop) {
  const int st = arena_get(slot, bytes, out);
  if (st != SIGMA_ERR_ALLOC) return st;
  drop();
  drop_optional_arenas();
  return arena_get(slot, bytes, out);
}

void set_last_error_text(const char* text);

// Functions run by sigma_shutdown() before the arenas are freed (plan caches).
typedef void (*ShutdownHook)();
void register_shutdown_hook(ShutdownHook h);

}  // namespace sigma
