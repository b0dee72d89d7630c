// FP64 discrete Fourier transforms as exact integer-digit products on the tensor cores (tcdft.cu).
#pragma once

#include "plan.h"

namespace sg {

struct ZInvArgs;
struct ZFwdArgs;
struct YArgs;
struct XArgs;
struct XNLArgs;

constexpr int kTcMaxJobs = 16;  // transforms per launch

// One column transform of a launch: out = factor * DFT^sign(in) over rows (row stride rs, in
// complex elements), factor taken from the table set; deriv = 1 first multiplies row k by i * k
// (k in [-n/2, n/2)), the table set's factor holding the wavenumber unit.
struct TcJob {
    const double2 *in;
    double2 *out;
    const double2 *add;   // added to the result when not null (same layout as out)
    const unsigned char *mat;  // matrix digits of the table set
    int deriv, expo;      // expo: power of two of the set's factor
    int prod;             // sums of products of physical rows: the first of the three derivatives' fields
    double post;          // further factor applied to the result (1: none)
    float top[2];         // sums of levels 3 and 4 that are smaller are exact (MatrixDigits)
};

// Columns: column c of a launch is at element (c / w) * s + c % w of a field, c in [0, ncol).
struct TcShape {
    int n, sign, nrows;         // nrows: rows of the result that are written
    int next;                   // rows [n - next, n) of the input are the FC-Gram continuation (0: none)
    unsigned ncol, w, s, rs;    // rs: row stride of in and out
    // transforms of rows: ncol rows; row r of tile t (128 rows) starts at t * ts + r * ls of the output
    unsigned ls;
    size_t ts;
};

// true when length n has digit-product transforms (FP64 plans)
bool tc_length_ok(int n);
// the table set of length n scaled by `factor` (half: for half spectra to real rows); built on first use
struct TcSet;
const TcSet *tc_set(Plan &P, int n, double factor, int *status, bool half = false);
void tc_job_set(TcJob &j, const TcSet *s);
// complex columns
int tc_run(Plan &P, const TcShape &s, const TcJob *jobs, int njobs, const char *name, double bytes);
// the passes of kernels.cuh over these transforms; kNoFast (fast.h) for a form that they do not take, and where
// their buffers or tables are not there and cannot be allocated
int tc_z_inverse(Plan &P, const ZInvArgs &a, int nf, double bytes);
int tc_z_forward(Plan &P, const ZFwdArgs &a, int nf, double bytes);
int tc_y(Plan &P, const YArgs &a, int nf, int nplanes, double bytes);
int tc_x(Plan &P, const XArgs &a, int nf, bool r2c, double bytes);
int tc_x_nonlinear(Plan &P, const XNLArgs &x, double bytes);
// the buffers of a solver's stage, allocated; kNoFast when there is no memory for them
int tc_reserve(Plan &P);
void tc_free(Plan &P);
unsigned long long tc_bytes(const Plan &P);
// An error when a kernel of the plan gave up a wait: its results are wrong, and so may be whatever was made of
// them.  Looked at before a transform is queued and wherever the plan's work has been waited for, so that no
// call that hands out results or reports completion succeeds after it.
int tc_status(const Plan &P);

}  // namespace sg
