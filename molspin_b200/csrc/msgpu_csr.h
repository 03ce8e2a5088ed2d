// msgpu_csr.h -- host passes over a Hamiltonian's CSR arrays (interleaved complex
// values).
#pragma once

#include <stddef.h>

#include <algorithm>
#include <cmath>
#include <vector>

namespace msgpu {

// Whether some row holds a column twice.  The column indices are in range.
inline bool repeated_columns(int dim, const int *rowptr, const int *col)
{
    std::vector<int> seen;  // last row that held a column; rows in ascending order need none
    for (int r = 0; r < dim; ++r) {
        bool ascending = true;
        for (int k = rowptr[r] + 1; k < rowptr[r + 1]; ++k) ascending = ascending && col[k] > col[k - 1];
        if (ascending) continue;
        if (seen.empty()) seen.assign(dim, -1);
        for (int k = rowptr[r]; k < rowptr[r + 1]; ++k) {
            if (seen[col[k]] == r) return true;
            seen[col[k]] = r;
        }
    }
    return false;
}

// The same matrices (nterms value arrays of rowptr[dim] entries on one pattern) with
// the entries of a row at one column added up, at the first one's place.
struct MergedCsr {
    std::vector<int> rowptr, col;
    std::vector<double> val;  // nterms x rowptr.back() complex
};
inline MergedCsr merge_columns(int dim, const int *rowptr, const int *col, const double *val, int nterms)
{
    MergedCsr out;
    out.rowptr.assign(1, 0);
    std::vector<int> row(dim, -1), at(dim, 0), to(rowptr[dim]);
    for (int r = 0; r < dim; ++r) {
        for (int k = rowptr[r]; k < rowptr[r + 1]; ++k) {
            if (row[col[k]] != r) {
                row[col[k]] = r;
                at[col[k]] = static_cast<int>(out.col.size());
                out.col.push_back(col[k]);
            }
            to[k] = at[col[k]];
        }
        out.rowptr.push_back(static_cast<int>(out.col.size()));
    }
    const size_t nnz = rowptr[dim], n = out.col.size();
    out.val.assign(2 * n * nterms, 0.0);
    for (int t = 0; t < nterms; ++t)
        for (size_t k = 0; k < nnz; ++k)
            for (int p = 0; p < 2; ++p) out.val[2 * (t * n + to[k]) + p] += val[2 * (t * nnz + k) + p];
    return out;
}

// Whether H's entries (one a column in each row) equal their transposes'
// conjugates to rounding: then, with K = kappa I, the Arnoldi matrix is
// tridiagonal and the three-term recurrence gives the same Krylov step.
inline bool is_hermitian(int dim, const int *rowptr, const int *col, const double *val)
{
    // rows are visited in order, so a sorted row's transposes come up in order too
    std::vector<int> next(rowptr, rowptr + dim);
    for (int r = 0; r < dim; ++r)
        for (int k = rowptr[r]; k < rowptr[r + 1]; ++k) {
            const int c = col[k];
            const double re = val[2 * static_cast<size_t>(k)], im = val[2 * static_cast<size_t>(k) + 1];
            const double tol = 4.0e-16 * (std::abs(re) + std::abs(im));
            auto conj_at = [&](int l) {
                return col[l] == r && std::abs(val[2 * static_cast<size_t>(l)] - re) <= tol &&
                       std::abs(val[2 * static_cast<size_t>(l) + 1] + im) <= tol;
            };
            if (next[c] < rowptr[c + 1] && conj_at(next[c])) {
                ++next[c];
                continue;
            }
            bool found = false;
            for (int l = rowptr[c]; l < rowptr[c + 1] && !found; ++l) found = conj_at(l);
            if (!found) return false;
        }
    return true;
}

// Largest absolute row sum.
inline double row_sum_norm(int dim, const int *rowptr, const double *val)
{
    double mx = 0.0;
    for (int r = 0; r < dim; ++r) {
        double s = 0.0;
        for (int k = rowptr[r]; k < rowptr[r + 1]; ++k)
            s += std::abs(val[2 * static_cast<size_t>(k)]) + std::abs(val[2 * static_cast<size_t>(k) + 1]);
        mx = std::max(mx, s);
    }
    return mx;
}

}  // namespace msgpu
