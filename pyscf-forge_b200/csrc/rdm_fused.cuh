// Fused RDM kernel (rdm_fused.cu), used by csffci_rdm12 and csffci_rdm12s.
#pragma once
#include "common.cuh"

namespace csffci {

// One Gram matrix over excitation rows of one or two row sets.
//   nsrc 1: M = X X^T of the set (both triangles filled)
//   nsrc 2: M[i][ld/2 + j] = X1_i . X2_j   (ld from rdm_fused_ld)
// sa: S/A rows (S first, A from rdm_fused_rows_s on; only S.S and A.A are
// formed), else the ordered rows T_pq, p*norb + q.  spin of a set: 1 alpha,
// 2 beta, 3 both.  sym (nsrc 1, sa): device flags of rdm_sym_check.
struct RdmFusedJob {
  int norb, nla, nlb, nsrc, sa;
  const csffci_link_t* la;
  const csffci_link_t* lb;
  const double* src[2];
  int spin[2];
  long long Na, Nb;
  const int* sym;
};

bool rdm_fused_fits(const RdmFusedJob& j);
// what its time depends on: output tiles of the Gram and passes over the
// determinants that they take, rows Ja and 16-column tiles of a CTA
struct RdmFusedSize {
  int out_tiles, passes;
  long long cta_rows, cta_tiles;
};
RdmFusedSize rdm_fused_size(const RdmFusedJob& j);
// workspace: partial sums, the matrix M with the two flags of rdm_sym_check
// behind its ld*ld elements, the packed beta links
size_t rdm_fused_workspace(int norb, long long Nb, int nlb);
double* rdm_fused_m(void* work);
int rdm_fused_ld(const RdmFusedJob& j);
int rdm_fused_rows_s(const RdmFusedJob& j);
int rdm_fused_run(const RdmFusedJob& j, void* work, cudaStream_t stream);
int rdm_sym_check(const double* c, long long n, int* bad, cudaStream_t stream);
int rdm_assemble_sa(const RdmFusedJob& j, const double* M, int nelec, double* dm1, double* dm2, cudaStream_t stream);
int rdm_assemble_sa_ab(const RdmFusedJob& j, const double* M, double* dm2, cudaStream_t stream);

}  // namespace csffci
