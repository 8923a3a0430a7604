/* emopt_modes.h -- device routines of the mode solver beside those of
 * emopt_fdtd.h (same library, same status codes). */
#ifndef EMOPT_MODES_H
#define EMOPT_MODES_H

#ifdef __cplusplus
extern "C" {
#endif

/* Inverses in place of the blocks W[lines[z]] (nb x nb complex128, row major),
 * z < nlines; info[z] (device) is 1 where a block is singular or not finite,
 * else 0.  work: device memory of FDTD_mode_invert_work(nb, nlines) bytes,
 * 256-byte aligned (0: a block of nb rows is too large for this routine).
 * Messages: FDTD_mode_last_error. */
long long FDTD_mode_invert_work(int nb, int nlines);
int FDTD_mode_invert(int nb, int device, void *stream, double *W, const int *lines, int nlines,
                     void *work, long long work_bytes, int *info);

#ifdef __cplusplus
}
#endif

#endif
