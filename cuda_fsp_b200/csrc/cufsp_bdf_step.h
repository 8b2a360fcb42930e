// cufsp_bdf_step.h -- one BDF step attempt as a single persistent launch (cufsp_bdf_step.cu).
#pragma once
#include "cufsp_internal.h"

namespace cufsp {

constexpr int kBdfHist = 8;   // difference history D_0..D_7
constexpr int kBdfOrder = 5;

struct BdfStepper;

// What the attempt needs of the integrator (device vectors of n doubles).
struct BdfStepIn {
    double *D[kBdfHist];
    double *w;              // error weights
    int k;                  // order
    double g[kBdfOrder + 1];  // g[j] = gamma_j, j >= 1
    double inv_alpha, c;    // 1 / alpha_k, h / alpha_k
    double econst;          // error constant of order k
    double atol, rtol, sqrt_n, eps_lin;
    const double *coefs;    // host: c_r(t_new)
    double *h_out;          // pinned host block of kBdfOutWords + 1 doubles, the sequence word that says when it
    unsigned *h_seq, *seq;  // has been written, and its counter
    double *d_out;          // not null: the launch reports into this device block, which is copied to h_out
};
constexpr int kBdfOutWords = 8;

enum BdfStepStatus { kBdfAccepted = 0, kBdfRejected = 1, kBdfNotConverged = 2, kBdfRhsNonfinite = 3,
                     kBdfBasisNonfinite = 4, kBdfErrNonfinite = 5 };
struct BdfStepOut {
    int status, iters;   // GMRES iterations
    double err;          // econst * ||d||_w
    double em, ep;       // ||D_k||_w, ||D_{k+2}||_w after an accepted step
};

// The stepper for a generator; *out = nullptr when the launch sequence is to be used (size or network out
// of range, CUFSP_BDF_PERSISTENT=0, or memory short).  Any other failure is an error, and the caller may ask
// again.
cufsp_status bdf_stepper_create(cufsp_mat *A, int maxl, cudaStream_t st, BdfStepper **out);
std::string bdf_stepper_describe(const BdfStepper *B);
void bdf_stepper_new_rates(BdfStepper *B);  // the rates to come are others: none has varied yet
void bdf_stepper_destroy(BdfStepper *B);
cufsp_status bdf_stepper_run(BdfStepper *B, const BdfStepIn &in, BdfStepOut &out, cudaStream_t st);

}  // namespace cufsp
