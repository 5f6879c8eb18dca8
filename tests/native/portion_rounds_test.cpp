// Rounds of chunks: every chunk once, a segment's in order, never more slots than there is room for; and as few rounds as the room allows.
#include <cstdio>
#include <cstdlib>
#include <random>

#include "portion_rounds.h"

static void require(bool ok, const char* what) {
  if (!ok) {
    std::printf("failed: %s\n", what);
    std::exit(1);
  }
}

template <int N> static int walk(const std::vector<int>& lens, int chunk, int from, size_t room, int few) {
  PortionRounds rounds(lens.data(), (int)lens.size(), chunk, from, room, few);
  std::vector<int> done(lens.size(), 0), place(lens.size(), -1);
  size_t chunks = 0;
  int count = 0, places = 0;
  for (int n : lens)
    if (n > 0 && n >= from) chunks += (n + chunk - 1) / chunk, ++places;
  require(rounds.places() == places, "places");
  const size_t most = rounds.slots();
  require(most <= std::max<size_t>(room, 1) && most <= chunks, "slots");
  PortionRound<N> r;
  while (rounds.next(r)) {
    ++count;
    require(r.items > 0 && r.items <= N && (size_t)r.slots <= most, "a round within the room");
    int slot = 0;
    for (int i = 0; i < r.items; ++i) {
      const PortionItem& p = r.item[i];
      require(p.slot == slot && p.count > 0, "slots in a row");
      slot += p.count;
      require(p.seg >= 0 && p.seg < (int)lens.size() && lens[p.seg] >= from, "who takes part");
      require(p.first == done[p.seg], "a segment from where its last round ended");
      done[p.seg] += p.count;
      require(p.place >= 0 && p.place < places && (place[p.seg] < 0 || place[p.seg] == p.place), "a place of its own");
      place[p.seg] = p.place;
    }
    require(slot == r.slots, "the slots in use");
  }
  for (size_t s = 0; s < lens.size(); ++s)
    require(done[s] == (lens[s] > 0 && lens[s] >= from ? (lens[s] + chunk - 1) / chunk : 0), "every chunk");
  return count;
}

int main() {
  std::vector<int> mixed(15, 32);
  mixed.push_back(2048);
  require(walk<32>(mixed, 64, 640, 79, 8) == 1, "short neighbours take no slots");              // 4 heads of 256 x 512 in 160 MB
  std::vector<int> delta(15, 32);
  delta.push_back(1531);
  require(walk<96>(delta, 16, 0, 234, 16) == 1, "nor more than they have blocks");                // 16 heads of 128 x 128 in 192 MB
  std::vector<int> many(63, 50);
  many.push_back(2048);
  require(walk<32>(many, 64, 640, 79, 8) == 1, "however many they are");
  require(walk<32>({2048, 2048, 2048, 2048}, 64, 640, 79, 8) == 2, "128 chunks through 79 slots");
  require(walk<32>(std::vector<int>(40, 2048), 64, 640, 79, 8) <= 20, "many long ones in groups");
  require(walk<2>({100, 100, 100}, 16, 0, 1000, 8) == 2, "no more items than a round holds");
  require(walk<32>({}, 64, 640, 79, 8) == 0 && walk<32>({639, 1}, 64, 640, 79, 8) == 0, "nobody");
  require(walk<32>({6400}, 64, 640, 0, 8) == 100, "one slot at least");
  std::mt19937 rng(1);
  for (int i = 0; i < 3000; ++i) {
    std::vector<int> lens(rng() % 40);
    for (int& n : lens) n = rng() % 3 ? rng() % 50 : rng() % 3000;
    const size_t room = rng() % 2 ? rng() % 20 : rng() % 300;
    const int few = 1 + rng() % 20, from = rng() % 2 ? 0 : rng() % 700, chunk = rng() % 2 ? 16 : 64;
    walk<32>(lens, chunk, from, room, few);
    walk<3>(lens, chunk, from, room, few);
  }
  std::printf("ok\n");
  return 0;
}
