// The shrink producers' allocation on the host, with the kernels' own rules: items of up to `rows_per_item` rows and eight
// tokens go through the ring one after the other, a stage is released no earlier than the producers have to wait for it.
// Prints one line per finding: two items whose last stages are in flight with the same reduction buffer, stages that
// overlap in the ring, a wait for a stage that has not been issued.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "lora_pipelined.cuh"

using namespace slora;

struct Stage {
  uint32_t off, size;
  long item;  // of a last stage, else -1
};

static int run(int h_in, int rows_per_item, const std::vector<std::pair<int, int>>& shapes, long items) {
  std::vector<Stage> stages;
  const uint32_t slots = shrink_slots(rows_per_item), buffers = shrink_buffers(rows_per_item);
  uint32_t tail = 0, head = 0;
  ItemEnds ends;
  int bad = 0;
  for (long item = 0; item < items && bad < 3; ++item) {
    const int nrows = shapes[item % shapes.size()].first, n = shapes[item % shapes.size()].second;
    const int kc = stage_k(nrows + n);
    for (int k0 = 0; k0 < h_in; k0 += kc) {
      const int klen = h_in - k0 < kc ? h_in - k0 : kc;
      const bool last = k0 + klen >= h_in;
      const uint32_t sz = round128(chunk_at(nrows + n, klen * 2)), released = ends.released(last, rows_per_item);
      const uint32_t g = static_cast<uint32_t>(stages.size());
      uint32_t at;
      while (!(ring_fits(head, tail == g, tail < g ? stages[tail].off : 0, kShrinkRingBytes, sz, at) && g - tail < slots &&
               tail >= released)) {
        if (tail == g) {
          printf("h_in %d rows %d: stage %u waits for itself\n", h_in, rows_per_item, g);
          return 1;
        }
        ++tail;
      }
      if (sz > static_cast<uint32_t>(kMaxStageBytes) || at + sz > static_cast<uint32_t>(kShrinkRingBytes)) {
        printf("h_in %d: %u bytes at %u\n", h_in, sz, at);
        ++bad;
      }
      head = at + sz;
      for (uint32_t s = tail; s < g; ++s) {
        if (stages[s].off < at + sz && at < stages[s].off + stages[s].size) {
          printf("h_in %d rows %d: stages %u and %u overlap\n", h_in, rows_per_item, s, g);
          ++bad;
        }
        if (last && stages[s].item >= 0 && stages[s].item % buffers == item % buffers) {
          printf("h_in %d rows %d: items %ld and %ld (%d rows, %d tokens) are both open in buffer %ld\n", h_in, rows_per_item,
                 stages[s].item, item, nrows, n, item % buffers);
          ++bad;
        }
      }
      stages.push_back({at, sz, last ? item : -1});
      if (last) ends.end_item(static_cast<uint32_t>(stages.size()));
    }
  }
  return bad;
}

int main() {
  static_assert(sizeof(ShrinkRed::sum) >= sizeof(float2) * 2 * kConsumerWarps * 64, "two buffers of sixteen rows");
  int bad = 0;
  for (int h_in : {8, 64, 520, 640, 1024, 1032, 1280, 1536, 1792, 2048, 2056, 2560, 3584, 4096, 5120, 5128, 8192, 16384}) {
    for (int rows_per_item : {4, 8, 16}) {
      // every shape by itself, then two that take turns and a shuffled row of all
      for (int nrows = 1; nrows <= rows_per_item; ++nrows)
        for (int n = 1; n <= 8; ++n) {
          bad += run(h_in, rows_per_item, {{nrows, n}}, 40);
          bad += run(h_in, rows_per_item, {{nrows, n}, {rows_per_item, 8}, {1, 1}}, 60);
        }
      srand(h_in * 31 + rows_per_item);
      std::vector<std::pair<int, int>> mixed;
      for (int i = 0; i < 2000; ++i) mixed.push_back({1 + rand() % rows_per_item, 1 + rand() % 8});
      bad += run(h_in, rows_per_item, mixed, 2000);
    }
  }
  printf(bad ? "%d findings\n" : "ok\n", bad);
  return bad != 0;
}
