// Prints, for a list of jobs (units and bytes each) on the command line, the
// batches that batch_units (eddy_host.cpp) makes of them: max_units max_bytes
// units bytes units bytes ... -> the batches' units, one a line.
#include <stdio.h>
#include <stdlib.h>

#include <vector>

#include "eddy_host.h"

int main(int argc, char **argv) {
  const int max_units = atoi(argv[1]);
  const size_t max_bytes = strtoull(argv[2], nullptr, 10);
  std::vector<eddy::BatchJob> jobs;
  for (int i = 3; i + 1 < argc; i += 2)
    jobs.push_back({atoi(argv[i]), (size_t)strtoull(argv[i + 1], nullptr, 10)});
  int job = 0, unit = 0;
  while (job < (int)jobs.size()) {
    const int n = eddy::batch_units(jobs, job, unit, max_units, max_bytes);
    if (n < 1) return 1;
    printf("%d\n", n);
    for (int left = n; left > 0;) {
      const int take = left < jobs[job].units - unit ? left : jobs[job].units - unit;
      left -= take;
      unit += take;
      if (unit == jobs[job].units) {
        job++;
        unit = 0;
      }
    }
  }
}
