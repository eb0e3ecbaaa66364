// knn_group_d4.cu -- the kNN kernel with a group of lanes per query, d = 4.
#include "ckd_knn_group.cuh"

namespace ckd {
CKD_KNN_GROUP(4)
}  // namespace ckd
