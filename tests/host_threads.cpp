// Work shared by threads of which only the calling one can be had: exit status 0 when all of it was done.
#include "../morello_b200/csrc/host_threads.hpp"
#include <atomic>
#include <cstdio>
#include <cstring>
#include <sys/resource.h>

int main(int argc, char** argv) {
  if (argc == 2 && !strcmp(argv[1], "none")) {   // no room for another thread's stack
    rlimit lim = {64 << 20, 64 << 20};
    if (setrlimit(RLIMIT_AS, &lim) != 0) return 2;
    rlimit stack = {512 << 20, 512 << 20};
    pthread_attr_t attr;
    pthread_attr_init(&attr);
    pthread_attr_setstacksize(&attr, stack.rlim_cur);
    if (pthread_setattr_default_np(&attr) != 0) return 2;
  }
  std::atomic<int> next{0}, helpers{0};
  int done[1000] = {};
  mrl::on_threads(4, [&](int t) {
    if (t) helpers++;
    for (int k = next++; k < 1000; k = next++) done[k]++;
  });
  for (int d : done) if (d != 1) return 1;
  printf("%d", helpers.load());
  return 0;
}
