// The small levels of a general 2x2-block FP64 V-cycle (tgmg.cu) in one launch
// over a cluster of blocks, in float pairs (mg_small_tg.cu): x periodic, y
// periodic or bounded, one Gauss-Seidel sweep down and one up per level, the
// coarsest level given as a matrix.  Coarse levels carry corrections, so the
// pairs' 2^-48 is relative to what the cycle still corrects.
#pragma once

#include <cuda_runtime.h>

#include <functional>
#include <vector>

namespace stzg {

// A level as the host set-up has it.
struct small_desc {
    int m, n;
    bool rows;             // the stencil depends on the row only
    const std::vector<int> *ids;  // stencil of every row (rows) or point
    bool ids_kept;                // the same as at the last setup
    std::vector<double> table;  // 40 doubles per stencil: nine blocks and the inverse centre
};

class small_cycle {
  public:
    // Lays out the levels first..ml of desc (bottom: the coarsest level's matrix,
    // 2mn x 2mn row-major) on stream st; ids must live until st is synchronised.
    // *moved is set where a launch captured before does not fit any more, also
    // when an error is returned.  active() tells whether the levels can be taken.
    int setup(const std::vector<small_desc> &desc, int yp, const std::vector<double> &bottom, cudaStream_t st,
              bool *moved);
    bool active() const { return t_ > 0; }
    int first() const { return t_; }  // its b and z are exchanged with launch's arrays
    void launch(const double2 *b, double2 *z, cudaStream_t st) const;
    ~small_cycle();

  private:
    struct buffer {
        void *p = nullptr;
        size_t cap = 0;
    };
    int need(buffer &b, size_t bytes, bool *moved);
    buffer tab_[17], cls_[17], dense_[17];
    std::vector<float4> pairs_[17];
    std::vector<float2> bottom_;
    std::vector<unsigned char> plan_;  // small_plan<ff>
    int t_ = 0, yp_ = 0;
};

}  // namespace stzg
