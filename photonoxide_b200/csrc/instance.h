// The library's internal view of one simulation context, for the batch (batch.cu), which steps
// several contexts' grids together in place: their device buffers, tables and sources as set.
#pragma once
#include <cuda_runtime.h>

#include <vector>

#include "common.cuh"
#include "photonoxide_fdtd.h"

struct InstanceView {
  int precision;
  int n[3];
  int pitch;  // values from a row of a y slab's psi to the next (n[0] padded)
  long long N;
  int periodic[3], low[3], high[3];
  double dt, step[3];
  double inv_step[3];  // 1/step as the kernels round it
  int fast_div[3];     // div_by_step's product form checked for the step
  int parity;  // which copy of E, H and H's psi is current
  void *e[2], *h[2], *psi_h[2], *psi_e;
  long long psi_h_len, psi_e_len;  // values in each copy of H's psi and in E's
  const void *ca;  // null: lossless
  const void *cb, *fe, *fh, *coefs;
  pxf::SlabEntry table[2][3][3][2];
  const std::vector<fdtd_waveform> *waves;
  const std::vector<fdtd_injection> *inj;
  long long nvalues;
  const long long *where;
  const pxf::SeriesDev *series;
  const long long *value_series;
  int nslots;
  const double *omega;
  const int *slot_field;
  double *sums;
  long long nsums;  // complex sums
  void *ring;  // the transforms' ring: ring_k rows of nvalues
  int ring_k;
  int freq_chunks;  // the most frequencies of a series, in chunks of DFT_F (at least 1)
  int nprobes;
  const long long *probes;
  bool media;
  bool plane_waves;  // total-field/scattered-field boxes (stepped by the engine alone)
  int naux;            // the values a step of its auxiliary runs records (te_block tiles only)
  cudaStream_t stream;
  unsigned long long layout;      // moves on with the calls that change what a batch's tables hold
  unsigned long long generation;  // moves on with every change the engine's calls make
};

int fdtd_instance_view(fdtd_ctx *c, InstanceView *v);
// The probe record's rows for `steps` more steps (grown as needed); null without probes.
int fdtd_instance_reserve(fdtd_ctx *c, long long steps, double **rows);
// After `steps` steps taken by the batch, the current copy having changed `flips` times: the
// current copies and the record's length.
void fdtd_instance_advance(fdtd_ctx *c, long long steps, int flips);
// `count` steps of the context's plane waves' auxiliary runs from step *base (device memory), their
// values into the tables of `stride` values a step after the emitters'; the kernels launched.
int fdtd_instance_aux(fdtd_ctx *c, int stride, const long long *base, int count, double *out_h,
                      double *out_e);
struct fdtd_batch;
// The batch takes a tile shape by its size alone, without timing any: one that is remade often.
void fdtd_batch_no_trial(fdtd_batch *batch);
// A 2D TE context's own steps on the batch's tiles of several steps a launch, enqueued on its stream
// (batch.cu). *batch: made on the first call, the context's to destroy. check: whether the fields may
// have come from elsewhere since the last such run: that H_x, H_y, E_z are zero is then looked up
// (and waited for); *te false: they are not, or it returns an error (its tables would take more than
// `room` bytes, or there is no memory for them), and nothing has run. rows: the probe record's (reserved);
// *held: the bytes its tables take. Adds its launches to *launches.
int fdtd_solo_run(fdtd_batch **batch, fdtd_ctx *c, bool check, int64_t steps, int64_t first,
                  double *rows, size_t room, size_t *held, bool *te, long long *launches);
// The transforms' sums since the last read added into `parts` (doubles, interleaved, laid end to
// end in the layout of fdtd_read_dft; lens: each part's), the device's then zero. Does nothing
// where no step has been taken since the last read. wide: a long read may be added by an OpenMP team;
// not in a thread that ends with the read, which would make and drop one.
int fdtd_instance_add_dft(fdtd_ctx *c, int nparts, double *const *parts, const long long *lens, bool wide);
int fdtd_instance_fail(fdtd_ctx *c, int code, const char *what);
