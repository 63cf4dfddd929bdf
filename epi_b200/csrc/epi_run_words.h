// Which device words the blocks of a resident run (epi_resident.cu) read and
// write between its grid barriers: plain index rules, shared with the host.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define EPI_HD __host__ __device__ __forceinline__
#else
#define EPI_HD inline
#endif

namespace epi {

// "Some tissue needs a candidate rebuild" in a run of steps. A step's commit
// raises it, and after the barrier that ends the step every block reads it
// and, if it is set, takes part in the rebuild that begins the next step. A
// fast block may commit the next step while a slow one has yet to read, so
// the word a step raises is never the one read at its beginning: gate is the
// word the run starts from (S.gate[0], which no step raises), step k raises
// words[k & 1]. A set word is cleared by one block within the rebuild it
// causes, past the rebuild's first barrier: by then every block has read it,
// and no block commits before the rebuild's last barrier. A word that is not
// set needs no clearing, so each is zero again when step k + 2 raises it.
struct RunFlags {
  int32_t* gate;
  int32_t* words;  // two, zero between runs
  EPI_HD int32_t* raised_by(int32_t step) const { return words + (step & 1); }
  EPI_HD int32_t* read_by(int32_t step) const { return step == 0 ? gate : raised_by(step - 1); }
  // After the last barrier, by one block (nobody else reads the words any
  // more), if the last step raised its word: the next run's first flag.
  EPI_HD void hand_on(int32_t nsteps) const {
    *read_by(nsteps) = 0;
    *gate = 1;
  }
};

// Barrier counts of runs that follow each other on a stream: two words, both
// zero at first. A run counts arrivals in its own, which must be zero when it
// starts, and clears the other for the next run as it starts itself. So the
// words change over only when a run was launched: after a refused launch the
// next run still finds the word that the last one cleared.
struct RunCount {
  uint32_t launched = 0;
  EPI_HD int own() const { return (int)(launched & 1u); }
  EPI_HD int next() const { return own() ^ 1; }
};

}  // namespace epi
