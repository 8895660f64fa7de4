// The plasticity update of FP32 and mixed storage on inverted particles whose F is near a
// reflection: F = U diag(s0, s1, -s2) V^T, where F^T F is as near to I as near a rotation.
// Prints "name value" pairs for strains 1e-7 to 0.2: the smallest det Re, the largest
// relative difference of Je and of Jp, and the largest difference of Fe and Re, the plastic
// update against the FP64 one on the same FP32 inputs; and for the non-plastic update the
// number of results that differ in any bit from the rotation U V^T of the FP32 SVD (mixed:
// refined once) and det F. Fe and Re are compared where the direction of the
// negative singular value is well determined: s2 at least 6e-4 below the others.
#include "mpm_math.cuh"
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>

using namespace mpm;

static void rotation(std::mt19937_64& g,double* R)
{
    std::normal_distribution<double> n(0.,1.);
    double w=n(g),x=n(g),y=n(g),z=n(g);
    const double s=1./std::sqrt(w*w+x*x+y*y+z*z);w*=s;x*=s;y*=s;z*=s;
    const double M[9]={1-2*(y*y+z*z),2*(x*y-w*z),2*(x*z+w*y),2*(x*y+w*z),1-2*(x*x+z*z),2*(y*z-w*x),2*(x*z-w*y),2*(y*z+w*x),1-2*(x*x+y*y)};
    std::memcpy(R,M,sizeof(M));
}
// max that keeps a NaN
static void worst(double& a,double b){if(!(b<=a)) a=b;}

template<class TS> static void family(const char* name,double strain,bool exact)
{
    const float cy=0.975f,sy=1.0075f;
    std::mt19937_64 g(5);
    std::uniform_real_distribution<double> u(0.,1.);
    double det=2,scalars=0,entries=0;int rotations=0;
    for(int it=0;it<5000;++it){
        double A[9],B[9],F[9];
        rotation(g,A);rotation(g,B);
        const double s[3]={exact?1.:1+strain*(.3+.7*u(g)),exact?1.:1+strain*(.3+.7*u(g)),exact?-1.:-(1-strain*(.3+.7*u(g)))};
        for(int i=0;i<3;++i) for(int j=0;j<3;++j) F[3*i+j]=A[3*i]*s[0]*B[3*j]+A[3*i+1]*s[1]*B[3*j+1]+A[3*i+2]*s[2]*B[3*j+2];
        if(exact&&it==0) for(int k=0;k<9;++k) F[k]=k==8?-1.:k%4==0?1.:0.;
        float Fm[9],Rm[9],lam,mu,Je,Jp=1.f;
        double Fx[9],Rx[9],lx,mx,Jx,Jq=1.;
        for(int k=0;k<9;++k){Fm[k]=(float)F[k];Fx[k]=Fm[k];}
        precompute<float,TS>(Fm,Jp,1e4f,2e4f,1,0.f,cy,sy,10.f,Rm,lam,mu,Je);
        precompute<double,double>(Fx,Jq,1e4,2e4,1,0.,(double)cy,(double)sy,10.,Rx,lx,mx,Jx);
        const double d=det3(Rm);
        if(!(d>=det)) det=d;
        worst(scalars,std::fabs(Je-Jx)/std::fabs(Jx));
        worst(scalars,std::fabs(Jp-Jq)/std::fabs(Jq));
        if(strain>=1e-3) for(int k=0;k<9;++k){worst(entries,std::fabs(Fm[k]-Fx[k]));worst(entries,std::fabs(Rm[k]-Rx[k]));}
        // not plastic
        float Fn[9],Rn[9],U[9],sv[3],V[9],W[9];
        for(int k=0;k<9;++k) Fn[k]=(float)F[k];
        svd3<float>(Fn,U,sv,V);
        mat_mul_bt(U,V,W);
        float Jn=1.f,J0=sv[0]*sv[1]*sv[2];
        if(sizeof(TS)==8){polar_refine_mixed(Fn,W);J0=det3_dot2(Fn);}
        precompute<float,TS>(Fn,Jn,1e4f,2e4f,0,0.f,cy,sy,10.f,Rn,lam,mu,Je);
        rotations+=std::memcmp(Rn,W,sizeof(W))!=0||Je!=J0;}
    std::printf("%s_det %.9g %s_scalars %.9g %s_entries %.9g %s_rotations %d ",name,det,name,scalars,name,entries,name,rotations);
}
int main()
{
    const struct {const char* name;double strain;} f[]={{"exact",0.},{"rigid",1e-7},{"light",1e-3},{"limit",0.007},{"far",0.2}};
    for(const auto& k:f){
        char n[32];
        std::snprintf(n,sizeof(n),"fp32_%s",k.name);family<float>(n,k.strain,k.strain==0.);
        std::snprintf(n,sizeof(n),"mixed_%s",k.name);family<double>(n,k.strain,k.strain==0.);}
    std::printf("\n");
    return 0;
}
