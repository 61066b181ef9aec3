// detected_lanes (csrc/lanes.h) on a buffer of exactly `lanes` entries that
// ends where an unreadable page begins (test infrastructure): a read past it
// ends the process. argv: lanes, every n-th lane detected; prints one mask a word.
#include <sys/mman.h>
#include <unistd.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "../../rrtl_gb300/csrc/lanes.h"

int main(int, char** argv) {
  const uint32_t lanes = (uint32_t)atoi(argv[1]), step = (uint32_t)atoi(argv[2]), words = (lanes + 31) / 32;
  const size_t page = (size_t)sysconf(_SC_PAGESIZE), bytes = (size_t)lanes * 4, room = (bytes + page - 1) / page * page;
  char* p = (char*)mmap(nullptr, room + page, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (p == MAP_FAILED || mprotect(p + room, page, PROT_NONE)) return 2;
  uint32_t* detect = (uint32_t*)(p + room - bytes);
  for (uint32_t l = 0; l < lanes; ++l) detect[l] = l % step ? 0xFFFFFFFFu : l;
  for (uint32_t w = 0; w < words + 3; ++w) printf("%u\n", rrtl::detected_lanes(detect, w, lanes));
  return 0;
}
