// C shim over the list of idle thread resources (bt-am_b200/csrc/idle_list.hpp),
// built with g++ for its CPU tests: resources are numbers, made and freed ones
// are counted.
#include "../../bt-am_b200/csrc/idle_list.hpp"

#include <atomic>

namespace {
struct Thing {
  int device = -1, id = -1;
};
struct Lot {
  btam::IdleList<Thing> list;
  std::atomic<int> made{0}, freed{0};
};
}  // namespace

extern "C" {
void *il_create() { return new Lot; }
void il_destroy(void *l) { delete static_cast<Lot *>(l); }
// the number of the thing, or -1; asked: the thread's count; fails: making fails
int il_acquire(void *p, int dev, int *asked, int fails) {
  Lot *l = static_cast<Lot *>(p);
  Thing t;
  const bool ok = l->list.acquire(dev, *asked, t, [&](Thing &r) {
    if (fails) return false;
    r.device = dev;
    r.id = l->made++;
    return true;
  });
  return ok ? t.id : -1;
}
void il_leave(void *p, int dev, int id) {
  Lot *l = static_cast<Lot *>(p);
  Thing t;
  t.device = dev;
  t.id = id;
  l->list.leave(t, [&](Thing &) { ++l->freed; });
}
void il_users(void *p, int by) {
  Lot *l = static_cast<Lot *>(p);
  l->list.users(by, [&](Thing &) { ++l->freed; });
}
int il_made(void *p) { return static_cast<Lot *>(p)->made; }
int il_freed(void *p) { return static_cast<Lot *>(p)->freed; }
int il_patience() { return btam::IdleList<Thing>::kPatience; }
int il_idle() { return (int)btam::IdleList<Thing>::kIdle; }
}
